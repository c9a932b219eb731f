// factor.cu -- the factored contraction of the chosen form.
//
// The R^k / S^k tables are sums of cell contributions (mrk_*/msk_*,
// dbsr_lib_dbs.f90:2898-3833): for electron-1 functions on interval iv and
// electron-2 functions on interval jv, a cell with iv < jv is the product of
// two 1-D moments, lo1(pair1,iv)*hi2(pair2,jv); iv > jv gives
// lo2(pair2,jv)*hi1(pair1,iv) (R^k only); iv == jv the diagonal-cell integral
// rkd.  A segment's density is a sum over its entries of orbital products,
// rho = sum_e c_e p1_{a_e} (x) p2_{b_e} with a_e, b_e the bound orbitals of
// K2, K3, so every contraction is linear in the ordered bound-orbital pairs
// (a,b).  The factored path therefore works per table with those pairs and
// per segment only with its coefficients:
//
// exchange (convol cases 3/4: R_data itype 4, S_data itypes 8/9), result
// out(x,y) over the output functions x, y of electrons 1 and 2:
//   far field |y-x| >= 9: every contributing cell has iv < jv, so
//     out = U C V^T with U_a(x) = sum_iv sum_x' lo1(x,x';iv) p_a(x'),
//     V_b(y) = sum_jv sum_y' hi2(y',y;jv) p_b(y') and C the segment's
//     coefficients over pairs (x-y >= 9: Ul C Vl^T, R^k only; zero for S^k);
//   near band |y-x| <= 8: out = sum_e c_e Kb_{a_e b_e}, where the band pair
//     potential Kb_ab(x,y) = sum_(i,j) W_xy(i,j) p1_a(i) p2_b(j) holds the
//     band-table element W_xy(i,j) that the exchange gather pairs with
//     density element (i,j) (built once per table, in two separable stages).
//
// direct (convol cases 1/2: R_data itype 3, S_data itypes 6/7): the band
// result is sum_e c_e Kd_{a_e b_e}, with the direct pair potential
//   Kd_ab(pair1) = sum_iv [lo1(pair1;iv) Suf_ab(iv) + hi1(pair1;iv) Pre_ab(iv)]
//                + sum_{pair2} rkd(pair1,pair2;iv) rho_ab(pair2)   (iv = jv)
// Suf/Pre the suffix/prefix sums over cells of the moment-weighted density of
// the pair, and rho_ab the pair density in the reference's storage (the
// symmetric 's' storage sums both orders, p1(f)p2(s)+p1(s)p2(f)).  Within the
// cells that an output belongs to, both terms are summed into one small matrix
// before any orbital is taken (k_pair_direct).
//
// The per-segment work is then a sum of a few dozen potential rows per
// output element, fused into the scatter for the direct cases.  All of this
// is FP64; with job.split the exchange far field runs as split-precision
// products on the tensor cores, fused with the near band and the scatter
// (exchange_tc.cu).
#include "internal.cuh"
#include "ff.cuh"
#include "pairs.cuh"

#include <algorithm>
#include <type_traits>

namespace {

constexpr int NB_MAX = 128;       // bound orbitals handled by the factored path
constexpr int FAR = 9;            // |y - x| >= FAR is far field (spline orders <= 9)
constexpr int BAND = FAR - 1;     // near band |y - x| <= 8
constexpr int NDB = 2 * BAND + 1; // band diagonals
constexpr int PXC = 4;            // output rows per block of the band pair potentials
constexpr int PDB = 32;           // second orbitals per block of the pair potentials
constexpr int PDT = 256;          // their threads

// target quadrants of the atypes of one list (UPDATE_HS)
struct QuadSpec {
  int na;
  int ii[4], jj[4];
};

// direct pair potentials of the atypes of one list (FP64, or float-float
// pairs in the split form)
struct KdSet {
  const double *K[4];
  const float2 *Kf[4];
};

// ---------------------------------------------------------------------------
// bound-orbital rows of both components (blockIdx.y):
// P[a*ns + x] = pq(x+1, comp, b2o[a]), and as float-float pairs
__global__ void k_bound_rows(int ns, int nb, const int *b2o, const double *pq, double *P,
                             float2 *Pf) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ns * nb) return;
  const int x = q % ns, a = q / ns, comp = blockIdx.y;
  const double v = pq[(size_t)x + (size_t)ns * comp + (size_t)2 * ns * (b2o[a] - 1)];
  const size_t o = (size_t)comp * ns * nb + q;
  P[o] = v;
  Pf[o] = ffa::split(v);
}

// ---------------------------------------------------------------------------
// far-field vectors of one electron: Ulo(x,a) = sum_xc tlo(x,xc) p_a(xc) (and Uhi
// with thi), x the output function, xc the contracted one, t the moments of the
// pair summed over its cells (k_moment_sums), and their float-float copies where
// asked for.  Both electrons' vectors (R^k: those of the P and Q pairs, which
// every type of the k shares) in one launch (blockIdx.y).  A thread takes the up
// to 2 ks - 1 functions xc, nine loads in flight.  ns 283, 20 orbitals: 8 us a k,
// 15.5 summing the cells of every pair for each orbital.
struct FarSide {
  int sym, out_first, ccomp;  // sym: t[min + ns |xc - x|], else t[first + ns (second - first + ks-1)]
  const double *tlo, *thi;
  double *Ulo, *Uhi;
  float2 *Flo, *Fhi;
};

__global__ void k_far_vectors(int ns, int ks, int nb, const int *b2o, const double *pq,
                              const FarSide s0, const FarSide s1) {
  const FarSide &sd = blockIdx.y ? s1 : s0;
  const int sym = sd.sym, out_first = sd.out_first, ccomp = sd.ccomp;
  const double *tlo = sd.tlo, *thi = sd.thi;
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ns * nb) return;
  const int x = q % ns, a = q / ns;  // 0-based
  const double *p = pq + (size_t)ns * (ccomp - 1) + (size_t)2 * ns * (b2o ? b2o[a] - 1 : a);
  double slo = 0.0, shi = 0.0;
  for (int d0 = 1 - ks; d0 < ks; d0 += 9) {
    double pv[9], lv[9], hv[9];
#pragma unroll
    for (int u = 0; u < 9; u++) {
      const int d = d0 + u, xc = x + d;
      const bool ok = d < ks && xc >= 0 && xc < ns;
      const int o = sym ? min(x, xc) + ns * abs(d)
                        : (out_first ? x + ns * (d + ks - 1) : xc + ns * (ks - 1 - d));
      pv[u] = ok ? p[xc] : 0.0;
      lv[u] = ok ? tlo[o] : 0.0;
      hv[u] = ok && thi ? thi[o] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 9; u++) {
      slo = fma(lv[u], pv[u], slo);
      shi = fma(hv[u], pv[u], shi);
    }
  }
  sd.Ulo[q] = slo;
  if (sd.Uhi) sd.Uhi[q] = shi;
  if (sd.Flo) sd.Flo[q] = ffa::split(slo);
  if (sd.Fhi) sd.Fhi[q] = ffa::split(shi);
}

// Z(a,y) = sum_{e in segment, first orbital a} c_e V(y, second orbital), also Zl with Vl
__global__ void k_far_z(int ns, int nb, const int *members, const SegInfo *info,
                        const int *pairs, const double *cd, const double *V, const double *Vl,
                        double *Z, double *Zl) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ns * nb) return;
  int a = q % nb, y = q / nb;
  int slot = blockIdx.y;
  SegInfo si = info[members[slot]];
  double z = 0.0, zl = 0.0;
  for (int e = si.start; e < si.end; e++) {
    const int pr = pairs[e];
    if (pr / nb != a) continue;
    const int b = pr - a * nb;
    z = fma(cd[e], V[(size_t)y + (size_t)ns * b], z);
    if (Vl) zl = fma(cd[e], Vl[(size_t)y + (size_t)ns * b], zl);
  }
  size_t o = (size_t)slot * nb * ns + q;  // Z[slot][a + nb*y]
  Z[o] = z;
  if (Zl) Zl[o] = zl;
}

// far field out(x,y) = U(x,:) Z(:,y) for y-x >= FAR, Ul(x,:) Zl(:,y) for
// x-y >= FAR; 32x32 output tiles, 256 threads with 4 outputs each, the
// orbital dimension staged through shared memory 32 at a time.
constexpr int FK = 32;
__global__ void __launch_bounds__(256) k_far_field(int ns, int nb, const double *U,
                                                   const double *Ul, const double *Z,
                                                   const double *Zl, double *Y, size_t per) {
  __shared__ double su[32][FK + 1], sz[FK][33];
  __shared__ double sul[32][FK + 1], szl[FK][33];
  const int slot = blockIdx.z;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  const bool any_up = (y0 + 31) - x0 >= FAR;
  const bool any_lo = Ul && (x0 + 31) - y0 >= FAR;
  if (!any_up && !any_lo) return;
  const double *Zs = Z + (size_t)slot * nb * ns;
  const double *Zls = Zl ? Zl + (size_t)slot * nb * ns : nullptr;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int a0 = 0; a0 < nb; a0 += FK) {
    const int na = min(FK, nb - a0);
    for (int q = threadIdx.x; q < 32 * FK; q += 256) {
      int r = q % 32, a = q / 32;
      int x = x0 + r, y = y0 + r;
      bool ok = a < na;
      su[r][a] = (ok && x < ns && any_up) ? U[(size_t)x + (size_t)ns * (a0 + a)] : 0.0;
      sz[a][r] = (ok && y < ns && any_up) ? Zs[(size_t)(a0 + a) + (size_t)nb * y] : 0.0;
      sul[r][a] = (ok && x < ns && any_lo) ? Ul[(size_t)x + (size_t)ns * (a0 + a)] : 0.0;
      szl[a][r] = (ok && y < ns && any_lo) ? Zls[(size_t)(a0 + a) + (size_t)nb * y] : 0.0;
    }
    __syncthreads();
    for (int t = 0; t < 4; t++) {
      int q = threadIdx.x + 256 * t;
      int r = q % 32, cc = q / 32;
      int d = (y0 + cc) - (x0 + r);
      double s = acc[t];
      if (d >= FAR)
        for (int a = 0; a < na; a++) s = fma(su[r][a], sz[a][cc], s);
      else if (d <= -FAR)
        for (int a = 0; a < na; a++) s = fma(sul[r][a], szl[a][cc], s);
      acc[t] = s;
    }
    __syncthreads();
  }
  double *Ys = Y + (size_t)slot * per;
  for (int t = 0; t < 4; t++) {
    int q = threadIdx.x + 256 * t;
    int r = q % 32, cc = q / 32;
    int x = x0 + r, y = y0 + cc;
    if (x >= ns || y >= ns) continue;
    int d = y - x;
    if (d >= FAR || (Ul && d <= -FAR)) Ys[(size_t)x + (size_t)ns * y] = acc[t];
  }
}

__host__ __device__ inline int pair_row_stride(int n) {  // 8 mod 16: rows on other banks
  return (n + 7) / 16 * 16 + 8;
}

// ---------------------------------------------------------------------------
// band pair potentials of an exchange table, one block per PXC output rows
// and one band diagonal d = y - x:
//   W(x; i, j)  the table element the exchange gather of output (x, y) pairs
//               with density element (i, j) (the gather of k_exchange in
//               assemble.cu, restricted to the band; every (i, j) meets one
//               element, so W needs no sums)
//   H(x; i, b)  = sum_j W(x; i, j) P2(b, j)
//   Kb(ab; x, y) = sum_i P1(a, i) H(x; i, b)
// mode 0: R table 's','s' case 3; 1: S 'n','n' case 3; 2: S 'n','n' case 4.
// Band table layout: rkb(i, j-i+BW+1, ip, jp) for |j - i| <= BW.
// FF: the table elements split into float-float pairs, both stages as
// float-float sums (ff.cuh), Kb written as float-float pairs (float2).
// Kx: where the results of the table with the electrons exchanged go, element
// (b a; y, x - y) for (a b; x, y - x).  R^k types 0 and 1 are unchanged under
// the exchange (Kx = Kout): only the diagonals d >= 0 are computed.  Type 2
// gives type 3's potentials this way (Kx theirs); S^k has none (Kx null).
// Positions past the ends of the grid are set to zero.
//
// PXC rows are a full sector of the results and of the table's rows; a block
// takes PDB second orbitals, a thread two of them at once, so that a value read
// from shared memory meets two sums.  Bound by the twelve FP32 instructions of a
// float-float multiply-add, otherwise by the FP64 pipe.  ns 283, 20 orbitals:
// 63 us a list in the mean over R^k and S^k; 86 us with one sum a thread (two
// loads a multiply-add), FP64 windows split by every block and a launch per
// table, and launches before to clear the results.
// The three tables of an R^k list are one launch (blockIdx.y: table and d), so
// that short grids fill the SMs too.
template <bool FF>
struct PairBandArgs {
  int ns, ks, nb, mode, bw;  // bw: stride of the second orbitals' arrays
  int y0[4];                 // first blockIdx.y of each table, and their end
  const double *rkb[3];
  const typename Val<FF>::T *P1[3], *P2[3];
  typename Val<FF>::T *Kout[3], *Kx[3];
};
constexpr int PBW = 2 * FAR - 1;         // window of one output, at most
constexpr int PBR = PXC - 1 + PBW;       // rows of a block's windows

template <bool FF>
__global__ void __launch_bounds__(PDT) k_pair_band(const PairBandArgs<FF> p) {
  using V = Val<FF>;
  using T = typename V::T;
  struct alignas(16) T2 {
    T a, b;
  };
  extern __shared__ __align__(16) unsigned char smband[];
  T *Wm = reinterpret_cast<T *>(smband);  // [PXC][PBW][PBW]: (i, j) at (i-x+ks-1, j-y+ks-1)
  const int bw = p.bw;
  T *H = Wm + PXC * PBW * PBW;            // [PXC][PBW][bw]
  T *p2w = H + PXC * PBW * bw;            // [PBR][bw]: P2(b, x0+d-(ks-1)+row)
  T *p1w = p2w + PBR * bw;                // [PBR][pstr]: P1(a, x0-(ks-1)+row)
  const int ns = p.ns, ks = p.ks, nb = p.nb, pstr = pair_row_stride(nb);
  const int W = 2 * ks - 1;               // offsets -(ks-1) .. ks-1
  const int x0 = blockIdx.x * PXC + 1;    // first output row (1-based)
  const int ty = ((int)blockIdx.y >= p.y0[1]) + ((int)blockIdx.y >= p.y0[2]);
  T *Kout = p.Kout[ty], *Kx = p.Kx[ty];
  const int d = (int)blockIdx.y - p.y0[ty] - (Kx == Kout ? 0 : BAND);
  const double *rkb = p.rkb[ty];
  const int zb = blockIdx.z * PDB, bc = min(PDB, nb - zb), ng = (bc + 1) / 2;
  const int kb = p.mode == 0 ? ks : W;
  constexpr int BW = DBSRG_TABLE_BAND, NJ = 2 * DBSRG_TABLE_BAND + 1;
  auto TB = [&](int i, int j, int ip, int jp) -> T {
    return V::of(rkb[(size_t)(i - 1) + (size_t)ns * ((size_t)(j - i + BW) +
               (size_t)NJ * ((size_t)(ip - 1) + (size_t)kb * (size_t)(jp - 1)))]);
  };
  for (int q = threadIdx.x; q < PXC * PBW * PBW; q += PDT) Wm[q] = V::zero();
  for (int q = threadIdx.x; q < PBR * nb; q += PDT) {
    const int a = q / PBR, r = q - a * PBR, x = x0 - (ks - 1) + r;
    p1w[r * pstr + a] = x >= 1 && x <= ns ? p.P1[ty][(size_t)a * ns + x - 1] : V::zero();
  }
  for (int q = threadIdx.x; q < PBR * bw; q += PDT) {
    const int b = q / PBR, r = q - b * PBR, y = x0 + d - (ks - 1) + r;
    p2w[r * bw + b] =
        b < bc && y >= 1 && y <= ns ? p.P2[ty][(size_t)(zb + b) * ns + y - 1] : V::zero();
  }
  __syncthreads();
  for (int q = threadIdx.x; q < PXC * kb * kb; q += PDT) {
    const int xl = q % PXC, r = q / PXC, ip = r % kb + 1, jp = r / kb + 1;
    const int x = x0 + xl, y = x + d;
    if (x > ns || y < 1 || y > ns) continue;
    T *w = Wm + (size_t)xl * PBW * PBW;
    auto put = [&](int i, int j, T v) { w[(i - x + ks - 1) * PBW + (j - y + ks - 1)] = v; };
    if (p.mode == 0) {
      if (y - jp + 1 >= 1 && x + ip - 1 <= ns)
        put(x + ip - 1, y - jp + 1, TB(x, y - jp + 1, ip, jp));
      if (ip > 1 && x - ip + 1 >= 1 && y - jp + 1 >= 1)
        put(x - ip + 1, y - jp + 1, TB(x - ip + 1, y - jp + 1, ip, jp));
      if (jp > 1 && x + ip - 1 <= ns && y + jp - 1 <= ns)
        put(x + ip - 1, y + jp - 1, TB(x, y, ip, jp));
      if (ip > 1 && jp > 1 && x - ip + 1 >= 1 && y + jp - 1 <= ns)
        put(x - ip + 1, y + jp - 1, TB(x - ip + 1, y, ip, jp));
    } else if (p.mode == 1) {
      const int j = y - jp + ks, ii = x + ip - ks;
      if (j < max(1, 1 + ks - jp) || j > min(ns, ns + ks - jp)) continue;
      if (x < max(1, 1 + ks - ip) || x > min(ns, ns + ks - ip)) continue;
      put(ii, j, TB(x, j, ip, jp));
    } else {
      const int i = x - ip + ks, jj = y + jp - ks;
      if (y < max(1, 1 + ks - jp) || y > min(ns, ns + ks - jp)) continue;
      if (i < max(1, 1 + ks - ip) || i > min(ns, ns + ks - ip)) continue;
      put(i, jj, TB(i, y, ip, jp));
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < PXC * W * ng; q += PDT) {
    const int r = q / ng, g = q - r * ng, xl = r / W, u = r - xl * W;
    const T *w = Wm + (xl * PBW + u) * PBW;
    const T *pp = p2w + xl * bw + 2 * g;
    V s0, s1;
    for (int v = 0; v < W; v++) {
      const T wv = w[v];
      const T2 b2 = *reinterpret_cast<const T2 *>(pp + v * bw);
      s0.mac(wv, b2.a);
      s1.mac(wv, b2.b);
    }
    *reinterpret_cast<T2 *>(H + (xl * PBW + u) * bw + 2 * g) = {s0.get(), s1.get()};
  }
  __syncthreads();
  const size_t per = (size_t)ns * NDB;
  const bool both = Kx && (Kx != Kout || d > 0);
  // items: xl fastest, then the first orbital, then the group of two second ones
  for (int q = threadIdx.x; q < PXC * nb * ng; q += PDT) {
    const int xl = q % PXC, r = q / PXC, g = r / nb, a = r - g * nb;
    const int x = x0 + xl, y = x + d, b = zb + 2 * g;
    if (x > ns) continue;
    V s0, s1;
    int xx = y;  // row of the exchanged element
    if (y >= 1 && y <= ns) {
      const T *pa = p1w + xl * pstr + a, *h = H + xl * PBW * bw + 2 * g;
      for (int u = 0; u < W; u++) {
        const T pv = pa[u * pstr];
        const T2 h2 = *reinterpret_cast<const T2 *>(h + u * bw);
        s0.mac(pv, h2.a);
        s1.mac(pv, h2.b);
      }
    } else {  // no element: as many are missing from the exchanged diagonal's other end
      const int m = abs(d);
      xx = m >= ns ? x : (d > 0 ? x - (ns - m) : x + (ns - m));
    }
    const size_t o = (size_t)(x - 1) + (size_t)ns * (d + BAND);
    const size_t ox = (size_t)(xx - 1) + (size_t)ns * (BAND - d);
    auto put = [&](int bb, T v) {
      Kout[((size_t)a * nb + bb) * per + o] = v;
      if (both) Kx[((size_t)bb * nb + a) * per + ox] = v;
    };
    put(b, s0.get());
    if (b + 1 < nb) put(b + 1, s1.get());
  }
}

// ---------------------------------------------------------------------------
// direct pair potentials.  ed: pairs of the density electron, eo: of the
// output electron.  Pair densities of a symmetric storage give every ordered
// (h1, h2) the moment of the unordered pair (pidx orders them).
//
// Pairs are numbered a + nb b, or, where exchanging the orbitals changes
// nothing (symab: packed symmetric density pairs of equal components), by the
// pairs a <= b alone, a + b (b + 1) / 2.
__host__ __device__ inline int pair_count(int nb, int symab) {
  return symab ? nb * (nb + 1) / 2 : nb * nb;
}
__device__ __forceinline__ int pair_number(int nb, int symab, int a, int b) {
  return a + (symab ? b * (b + 1) / 2 : b * nb);
}

// The potentials of up to four tables (an R^k list's types) are built together:
// one launch of each of the three kernels.  ns 80, 5 orbitals: k_pair_direct 4 x 18
// -> 23 us, the three kernels of a list about 143 -> 40; energy functional, ns 300,
// 30 orbitals: 312 -> 249 us a multipole (6.2 -> 5.4 ms).
struct PairCellArgs {
  PairSpec ed[4];
  int symab[4];
  const double *M1[4], *M2[4], *P1[4], *P2[4];
  double *S1[4], *S2[4];  // S2 (with M2): null where one field only
};

// (1) cell sums, one block per cell cv and table:
//   S1(cv, pair) = sum_{h1,h2} M1(h1,h2;cv) P1(a, cv+h1-1) P2(b, cv+h2-1), S2 with M2
__global__ void k_pair_cellsum(int ns, int kk, int nb, const PairCellArgs g) {
  const int ty = blockIdx.y, symab = g.symab[ty];
  const PairSpec ed = g.ed[ty];
  const double *M1 = g.M1[ty], *M2 = g.M2[ty], *P1 = g.P1[ty], *P2 = g.P2[ty];
  double *S1 = g.S1[ty], *S2 = g.S2[ty];
  extern __shared__ double sm[];
  const int cv = blockIdx.x + 1, k1 = ed.k1, k2 = ed.k2;
  double *w1 = sm, *w2 = w1 + nb * k1, *t1 = w2 + nb * k2, *t2 = t1 + nb * k1;
  for (int q = threadIdx.x; q < nb * k1; q += blockDim.x) {
    const int a = q / k1, x = cv + q % k1;
    w1[q] = x <= ns ? P1[(size_t)a * ns + x - 1] : 0.0;
  }
  for (int q = threadIdx.x; q < nb * k2; q += blockDim.x) {
    const int b = q / k2, x = cv + q % k2;
    w2[q] = x <= ns ? P2[(size_t)b * ns + x - 1] : 0.0;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nb * k1; q += blockDim.x) {
    const int b = q / k1, h1 = q % k1 + 1;
    double s1 = 0.0, s2 = 0.0;
    for (int h2 = 1; h2 <= k2; h2++) {
      const size_t o = (size_t)pidx(ed, h1, h2) + (size_t)kk * (cv - 1);
      const double p = w2[b * k2 + h2 - 1];
      s1 = fma(M1[o], p, s1);
      if (M2) s2 = fma(M2[o], p, s2);
    }
    t1[q] = s1;
    t2[q] = s2;
  }
  __syncthreads();
  const int np = pair_count(nb, symab);
  for (int q = threadIdx.x; q < np; q += blockDim.x) {
    int a, b;
    if (symab) {
      b = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
      while (b * (b + 1) / 2 > q) b--;
      while ((b + 1) * (b + 2) / 2 <= q) b++;
      a = q - b * (b + 1) / 2;
    } else {
      b = q / nb;
      a = q - b * nb;
    }
    double s1 = 0.0, s2 = 0.0;
    for (int h = 0; h < k1; h++) {
      const double p = w1[a * k1 + h];
      s1 = fma(p, t1[b * k1 + h], s1);
      if (M2) s2 = fma(p, t2[b * k1 + h], s2);
    }
    S1[(size_t)(cv - 1) * np + q] = s1;
    if (M2) S2[(size_t)(cv - 1) * np + q] = s2;
  }
}

// (2) exclusive suffix (sum over later cells) or prefix sums per pair, in place:
// eight pairs a block, each with sixteen runs of cells (blockIdx.y: twice the
// table, odd ones its second array, prefix sums).  Bound by the FP64
// instructions, so the pairs are spread over many blocks: an R^k list's four
// tables at ns 300, 30 orbitals 16.5 us.
constexpr int PSW = 16, PSP = 8;
struct PairScanArgs {
  int np[4], suffix0[4];
  double *S[4][2];
};
__global__ void __launch_bounds__(PSP * PSW) k_pair_scan(int nv, const PairScanArgs g) {
  __shared__ double tot[PSW][PSP];
  const int lane = threadIdx.x % PSP, w = threadIdx.x / PSP, q = blockIdx.x * PSP + lane;
  const int ty = blockIdx.y / 2, which = blockIdx.y % 2, np = g.np[ty];
  if (!g.S[ty][which]) return;
  double *s = g.S[ty][which] + q;
  const bool suf = which == 0 && g.suffix0[ty], ok = q < np;
  const int run = (nv + PSW - 1) / PSW, lo = min(nv, w * run), hi = min(nv, lo + run);
  double t = 0.0;
  if (ok)
#pragma unroll 8
    for (int i = lo; i < hi; i++) t += s[(size_t)(suf ? hi - 1 - (i - lo) : i) * np];
  tot[w][lane] = t;
  __syncthreads();
  if (!ok) return;
  double acc = 0.0;
  if (suf)
    for (int k = PSW - 1; k > w; k--) acc += tot[k][lane];
  else
    for (int k = 0; k < w; k++) acc += tot[k][lane];
  // (loads of eight cells before their stores: the array is overwritten)
  for (int i0 = lo; i0 < hi; i0 += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + u;
      v[u] = i < hi ? s[(size_t)(suf ? hi - 1 - (i - lo) : i) * np] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + u;
      if (i >= hi) break;
      s[(size_t)(suf ? hi - 1 - (i - lo) : i) * np] = acc;
      acc += v[u];
    }
  }
}

// (3) the potentials.  An output (f, f+dl) belongs to the cells lo .. hi that
// hold both functions.  Everything the density does inside those cells goes
// through one small matrix per output, the table's elements without the far
// cells,
//   W(x,y) = sum_cv [ R(po(cv); x,y; cv) + M1(x,y;cv) sum_{cv' before} L1(po(cv'))
//                     + M2(x,y;cv) sum_{cv' after} L2(po(cv')) ],
// (x, y within the cells' functions, at most 17 x 17 at order 9, banded), and
//   Kd_ab = sum_x P1_a(x) H_b(x) + SA_ab sum_cv L1 + SB_ab sum_cv L2,
//   H_b(x) = sum_y W(x,y) P2_b(y),
// with SA/SB the scanned sums beyond the window (L1 = lo1, SA after the window;
// case 2: L1 = hi2, SA before it and the sum over cv' after).  Those two terms are
// FP64 in both forms: their factors, sums of r^k and of r^-(k+1), need its
// exponents (first cell of a grid to 1e-4, k = 11: 1e45 and less than 1e-45),
// their products do not.  As float-float pairs they took 72 us a list at ns 283
// and 96 at ns 400, 20 orbitals (81 and 109 in FP64), and gave NaN there.  Per pair an
// output takes up to 17 + 2 multiply-adds; contracting every diagonal cell by
// itself and adding the separable terms cell by cell takes up to 81 + 18.
// A block forms PDX consecutive f (a full sector of the result) of one dl
// for PDB second orbitals; a thread takes two second orbitals at once.  The
// small matrix is summed in FP64 and rebuilt by every block, so blocks of 16
// second orbitals lose more than they gain (106 us for 78).  Bound by the FP64
// pipe, in the split form by the latency of the small matrix's loads.  Cell by
// cell with partial sums in memory against this: ns 300, 30 orbitals, R^k, FP64
// 325 -> 78 us; ns 400, 20 orbitals, split form (R^k and S^k) 217 -> 55 us.
constexpr int PDX = 4;
template <bool FF>
struct PairDirTable {
  int np, symab, suf;
  PairSpec eo, ed;
  const double *rkd;  // element (po, pd; cell) at rpo po + rpd pd + rcell cell
  size_t rcell;
  int rpo, rpd;
  const double *L1, *L2, *M1, *M2, *SA, *SB;
  const typename Val<FF>::T *P1, *P2;
  typename Val<FF>::T *K;
};
template <bool FF>
struct PairDirArgs {
  int ns, nv, kk, nb, ncol, dl0;  // dl0: dl of column 0
  int bw;                         // stride of the second orbitals' arrays
  size_t per;
  PairDirTable<FF> t[4];          // blockIdx.y: table ncol + column
};

// KM: the largest spline order the shared arrays are laid out for (9, or 16 for
// the orders above: the energy functional takes them all)
constexpr int pair_window(int km) { return 2 * km - 1; }
constexpr int pair_rows(int km) { return PDX - 1 + pair_window(km); }

template <bool FF, int KM>
__global__ void __launch_bounds__(PDT) k_pair_direct(const PairDirArgs<FF> g) {
  const PairDirTable<FF> &p = g.t[blockIdx.y / g.ncol];
  constexpr int PDW = pair_window(KM), PDR = pair_rows(KM);
  using V = Val<FF>;
  using T = typename V::T;
  struct alignas(16) T2 {
    T a, b;
  };
  extern __shared__ __align__(16) unsigned char smdir[];
  T *W = reinterpret_cast<T *>(smdir);     // [PDX][PDW][PDW]
  const int bw = g.bw;
  T *H = W + PDX * PDW * PDW;              // [PDX][PDW][bw]
  T *p2w = H + PDX * PDW * bw;             // [PDR][bw]
  T *p1w = p2w + PDR * bw;                 // [PDR][pstr]
  __shared__ double c1[PDX][KM], c2[PDX][KM], t1[PDX], t2[PDX];
  __shared__ int los[PDX], his[PDX], pos[PDX][KM];
  const size_t per = g.per;
  const int ns = g.ns, nb = g.nb, kk = g.kk, pstr = pair_row_stride(nb);
  const PairSpec eo = p.eo, ed = p.ed;
  const int f0 = blockIdx.x * PDX + 1, col = blockIdx.y % g.ncol, dl = g.dl0 + col, zb = blockIdx.z * PDB;
  const int bc = min(PDB, nb - zb), na = p.symab ? zb + bc : nb;
  const int rb = f0 + max(1 - eo.k1, dl + 1 - eo.k2);  // first row of the windows
  if (threadIdx.x < PDX) {
    const int fl = threadIdx.x, f = f0 + fl, s2 = f + dl;
    int lo = max(1, rb + fl), hi = min(g.nv, min(f, s2));
    if (f > ns || s2 < 1 || s2 > ns) hi = lo - 1;
    double l1[KM], l2[KM], s1 = 0.0, s2s = 0.0;
#pragma unroll
    for (int k = 0; k < KM; k++) {
      const int cv = lo + k;
      const bool ok = cv <= hi;
      const int po = ok ? pidx(eo, f - cv + 1, s2 - cv + 1) : 0;
      const size_t o = (size_t)po + (size_t)kk * (ok ? cv - 1 : 0);
      l1[k] = ok ? p.L1[o] : 0.0;
      l2[k] = ok && p.L2 ? p.L2[o] : 0.0;
      pos[fl][k] = po;
    }
    // sums over the window's cells before (c1 where suf) or after a cell
#pragma unroll
    for (int k = 0; k < KM; k++) {
      if (p.suf) c1[fl][k] = s1;
      s1 += l1[k];
    }
    double r1 = 0.0;
#pragma unroll
    for (int k = KM - 1; k >= 0; k--) {
      c2[fl][k] = s2s;
      s2s += l2[k];
      if (!p.suf) c1[fl][k] = r1;
      r1 += l1[k];
    }
    t1[fl] = s1;
    t2[fl] = s2s;
    los[fl] = lo;
    his[fl] = hi;
  }
  for (int q = threadIdx.x; q < PDR * na; q += PDT) {
    const int a = q / PDR, r = q - a * PDR, x = rb + r;
    p1w[r * pstr + a] = x >= 1 && x <= ns ? p.P1[(size_t)a * ns + x - 1] : V::zero();
  }
  for (int q = threadIdx.x; q < PDR * bw; q += PDT) {
    const int b = q / PDR, r = q - b * PDR, y = rb + r;
    p2w[r * bw + b] =
        b < bc && y >= 1 && y <= ns ? p.P2[(size_t)(zb + b) * ns + y - 1] : V::zero();
  }
  __syncthreads();
  // one item per element, diagonal by diagonal (symmetric: the upper ones)
  const int u0 = ed.sym ? 0 : 1 - ed.k1, ndg = ed.k2 - u0;
  for (int q = threadIdx.x; q < PDX * PDW * ndg; q += PDT) {
    const int r = q / PDW, t = q - r * PDW, fl = r % PDX, u = t + u0 + r / PDX;
    const int lo = los[fl], hi = his[fl], x = lo + t, y = lo + u;
    const int ca = max(lo, max(x - ed.k1, y - ed.k2) + 1), cb = min(hi, min(x, y));
    if (ca > cb) continue;
    double v = 0.0;
#pragma unroll 9
    for (int cv = ca; cv <= cb; cv++) {
      const int pd = pidx(ed, x - cv + 1, y - cv + 1);
      const size_t o = (size_t)pd + (size_t)kk * (cv - 1);
      v += p.rkd[p.rcell * (cv - 1) + (size_t)p.rpo * pos[fl][cv - lo] +
                 (size_t)p.rpd * pd];
      v = fma(p.M1[o], c1[fl][cv - lo], v);
      if (p.M2) v = fma(p.M2[o], c2[fl][cv - lo], v);
    }
    const T wv = V::of(v);
    W[(fl * PDW + t) * PDW + u] = wv;
    if (ed.sym) W[(fl * PDW + u) * PDW + t] = wv;
  }
  __syncthreads();
  const int ng = (bc + 1) / 2;  // groups of two second orbitals
  for (int q = threadIdx.x; q < PDX * PDW * ng; q += PDT) {
    const int r = q / ng, g = q - r * ng, fl = r / PDW, t = r - fl * PDW;
    const int lo = los[fl], hi = his[fl], x = lo + t;
    const int ca = max(lo, x - ed.k1 + 1), cb = min(hi, x);
    if (ca > cb) continue;
    const T *w = W + r * PDW;
    const T *pp = p2w + (lo - rb) * bw + 2 * g;
    V s0, s1;
    for (int u = ca - lo; u < cb + ed.k2 - lo; u++) {
      const T wv = w[u];
      const T2 v = *reinterpret_cast<const T2 *>(pp + u * bw);
      s0.mac(wv, v.a);
      s1.mac(wv, v.b);
    }
    *reinterpret_cast<T2 *>(H + r * bw + 2 * g) = {s0.get(), s1.get()};
  }
  __syncthreads();
  // items: fl fastest, then the first orbital, then the group
  const int nitem = p.symab ? ng * zb + ng * (ng + 1) : ng * na;
  for (int q = threadIdx.x; q < PDX * nitem; q += PDT) {
    const int fl = q % PDX, f = f0 + fl;
    int a = q / PDX, g = 0;
    if (p.symab) {  // group g holds the first orbitals up to its second one
      while (a >= zb + 2 * g + 2) a -= zb + 2 * g + 2, g++;
      if (a >= na) continue;
    } else {
      g = a / na;
      a -= g * na;
    }
    if (f > ns) continue;
    const int lo = los[fl], hi = his[fl], b0 = zb + 2 * g;
    V s0, s1;
    Val<false> far0, far1;
    if (lo <= hi) {
      const T *pa = p1w + (lo - rb) * pstr + a, *h = H + fl * PDW * bw + 2 * g;
      const int nt = hi - lo + ed.k1;
      for (int t = 0; t < nt; t++) {
        const T pv = pa[t * pstr];
        const T2 v = *reinterpret_cast<const T2 *>(h + t * bw);
        s0.mac(pv, v.a);
        s1.mac(pv, v.b);
      }
      const size_t ra = (size_t)((p.suf ? hi : lo) - 1) * p.np, rl = (size_t)(lo - 1) * p.np;
      const int q0 = pair_number(nb, p.symab, p.symab ? min(a, b0) : a, b0);
      const int q1 = pair_number(nb, p.symab, a, min(b0 + 1, nb - 1));
      if constexpr (!FF) far0.v = s0.v, far1.v = s1.v;
      far0.mac(t1[fl], p.SA[ra + q0]);
      far1.mac(t1[fl], p.SA[ra + q1]);
      if (p.SB) {
        far0.mac(t2[fl], p.SB[rl + q0]);
        far1.mac(t2[fl], p.SB[rl + q1]);
      }
      if constexpr (FF) {
        far0.v += s0.value();
        far1.v += s1.value();
      }
    }
    const size_t o = (size_t)(f - 1) + (size_t)ns * col;
    auto put = [&](int b, T v) {
      p.K[((size_t)a * nb + b) * per + o] = v;
      if (p.symab && a < b) p.K[((size_t)b * nb + a) * per + o] = v;
    };
    if (!p.symab || a <= b0) put(b0, V::of(far0.v));
    if (b0 + 1 < nb) put(b0 + 1, V::of(far1.v));
  }
}

// ---------------------------------------------------------------------------
// near band of the exchange results: Y(x, x+d) = sum_e c_e Kb(pair_e; x, d)
__global__ void k_band_sum(int ns, const int *members, const SegInfo *info, const int *pairs,
                           const double *cd, const double *Kb, double *Y, size_t per) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ns * NDB) return;
  const int slot = blockIdx.y;
  const int x = t % ns + 1, y = x + t / ns - BAND;
  if (y < 1 || y > ns) return;
  const SegInfo si = info[members[slot]];
  const size_t kper = (size_t)ns * NDB;
  double acc = 0.0;
  for (int e = si.start; e < si.end; e++) acc = fma(cd[e], Kb[(size_t)pairs[e] * kper + t], acc);
  Y[(size_t)slot * per + (size_t)(x - 1) + (size_t)ns * (y - 1)] = acc;
}

// Exchange scatter (UPDATE_HS, updates.f90:110-179): one 32x32 tile of one
// quadrant of an owner's block; contributions in the reference's order
// (atype-major, owner then partner), transposed reads staged through shared
// memory so that every global access is coalesced.  Without a lower far
// field (S^k) the region x - y >= 9 of every result is zero.
__global__ void __launch_bounds__(256) k_scatter_x(int ns, QuadSpec sp, int nm,
                                                   const int *members, const int *own_slots,
                                                   const SegInfo *info, const double *Y,
                                                   int lower, double *hch) {
  __shared__ double tt[32][33];
  const int ms = 2 * ns, nt = (ns + 31) / 32;
  const int quad = blockIdx.x / (nt * nt), tile = blockIdx.x % (nt * nt);
  const int qr = quad % 2 + 1, qc = quad / 2 + 1;
  const int r0 = (tile % nt) * 32, c0 = (tile / nt) * 32;
  const int oslot = own_slots[blockIdx.y];
  const SegInfo si = info[members[oslot]];
  if (si.blk < 1) return;
  const int pslot = si.partner >= 0 ? oslot + 1 : -1;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  const size_t per = (size_t)ns * ns;
  double *hb = hch + (size_t)(si.blk - 1) * ms * ms + (size_t)(qr - 1) * ns + (size_t)ms * (qc - 1) * ns;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  bool touched = false;
  for (int a = 0; a < sp.na; a++) {
    for (int pass = 0; pass < 2; pass++) {
      const int slot = pass == 0 ? oslot : pslot;
      if (slot < 0) break;
      const SegInfo sj = info[members[slot]];
      const double *d = Y + ((size_t)a * nm + slot) * per;
      const int ii = sp.ii[a], jj = sp.jj[a];
      const bool eq = sj.ich == sj.jch;
      const bool dir = (sj.ich > sj.jch || eq) && qr == ii && qc == jj;
      const bool tra = (sj.ich < sj.jch && qr == ii && qc == jj) || (eq && qr == jj && qc == ii);
      if (!dir && !tra) continue;
      if (!touched) {
        touched = true;
        for (int k = 0; k < 4; k++) {
          const int lr = r0 + tx, lc = c0 + ty + 8 * k;
          if (lr < ns && lc < ns) v[k] = hb[(size_t)lr + (size_t)ms * lc];
        }
      }
      if (dir) {
        for (int k = 0; k < 4; k++) {
          const int lr = r0 + tx, lc = c0 + ty + 8 * k;
          if (lr >= ns || lc >= ns) continue;
          const double y = (lower || lr - lc < FAR) ? d[(size_t)lr + (size_t)ns * lc] : 0.0;
          v[k] = v[k] + (eq ? y / 2.0 : y);
        }
      }
      if (tra) {
        __syncthreads();
        for (int k = 0; k < 4; k++) {
          const int x = c0 + tx, y = r0 + ty + 8 * k;  // y(x, y) = element (lc, lr)
          tt[ty + 8 * k][tx] =
              (x < ns && y < ns && (lower || x - y < FAR)) ? d[(size_t)x + (size_t)ns * y] : 0.0;
        }
        __syncthreads();
        for (int k = 0; k < 4; k++) {
          const int lr = r0 + tx, lc = c0 + ty + 8 * k;
          if (lr >= ns || lc >= ns) continue;
          const double y = tt[tx][ty + 8 * k];
          v[k] = v[k] + (eq ? y / 2.0 : y);
        }
      }
    }
  }
  if (!touched) return;
  for (int k = 0; k < 4; k++) {
    const int lr = r0 + tx, lc = c0 + ty + 8 * k;
    if (lr < ns && lc < ns) hb[(size_t)lr + (size_t)ms * lc] = v[k];
  }
}

// position of element (i, j) (1-based) of the band result y in its ns x ncol
// storage, or -1 where the storage holds no element (yval of assemble.cu)
__device__ __forceinline__ int band_pos(int ns, int ks, char sym, int i, int j) {
  if (sym == 's') {
    const int lo = min(i, j), dl = abs(i - j);
    return dl >= ks ? -1 : (lo - 1) + ns * dl;
  }
  const int jp = j - i + ks;
  return (jp < 1 || jp > 2 * ks - 1) ? -1 : (i - 1) + ns * (jp - 1);
}

// Direct scatter: every band element of the four quadrants of an owner's
// block; each contribution is formed from the pair potentials and the
// segment's coefficients where it is added (FF: as a float-float sum).
template <bool FF>
__global__ void k_scatter_dp(int ns, int ks, char sym, QuadSpec sp, KdSet kd,
                             const int *members, const int *own_slots, const SegInfo *info,
                             const int *pairs, const double *cd, const float2 *cdf,
                             double *hch) {
  const int ms = 2 * ns, nd = 2 * ks - 1;
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (size_t)4 * ns * nd) return;
  const int oslot = own_slots[blockIdx.y];
  const SegInfo si = info[members[oslot]];
  if (si.blk < 1) return;
  const int pslot = si.partner >= 0 ? oslot + 1 : -1;
  const int quad = (int)(q / ((size_t)ns * nd));
  const int rem = (int)(q % ((size_t)ns * nd));
  const int lr = rem % ns, lc = lr + rem / ns - (ks - 1);
  if (lc < 0 || lc >= ns) return;
  const int qr = (quad & 1) + 1, qc = (quad >> 1) + 1;
  const size_t per = (size_t)ns * (sym == 's' ? ks : nd);
  double *h = hch + (size_t)(si.blk - 1) * ms * ms + (size_t)((qr - 1) * ns + lr) +
              (size_t)ms * ((qc - 1) * ns + lc);
  bool touched = false;
  double val = 0.0;
  auto ysum = [&](int a, const SegInfo &sj, int i, int j) -> double {
    const int p = band_pos(ns, ks, sym, i, j);
    if (p < 0) return 0.0;
    // entries in batches of EB: the EB potential loads are issued together
    // (they depend only on the batch's pair indices), then summed in order
    constexpr int EB = 8;
    int e = sj.start;
    if (FF) {
      const float2 *K = kd.Kf[a];
      float sh = 0.0f, sl = 0.0f;
      for (; e + EB <= sj.end; e += EB) {
        float2 kv[EB];
#pragma unroll
        for (int u = 0; u < EB; u++) kv[u] = K[(size_t)pairs[e + u] * per + p];
#pragma unroll
        for (int u = 0; u < EB; u++) ffa::mac(cdf[e + u], kv[u], sh, sl);
        // the low sum back below half an ulp of the high one, so that its own
        // rounding does not grow with the entries
        const float2 r = ffa::norm(sh, sl);
        sh = r.x;
        sl = r.y;
      }
      for (; e < sj.end; e++) ffa::mac(cdf[e], K[(size_t)pairs[e] * per + p], sh, sl);
      return ffa::value(sh, sl);
    }
    const double *K = kd.K[a];
    double acc = 0.0;
    for (; e + EB <= sj.end; e += EB) {
      double kv[EB];
#pragma unroll
      for (int u = 0; u < EB; u++) kv[u] = K[(size_t)pairs[e + u] * per + p];
#pragma unroll
      for (int u = 0; u < EB; u++) acc = fma(cd[e + u], kv[u], acc);
    }
    for (; e < sj.end; e++) acc = fma(cd[e], K[(size_t)pairs[e] * per + p], acc);
    return acc;
  };
  for (int a = 0; a < sp.na; a++) {
    for (int pass = 0; pass < 2; pass++) {
      const int slot = pass == 0 ? oslot : pslot;
      if (slot < 0) break;
      const SegInfo sj = info[members[slot]];
      const int ii = sp.ii[a], jj = sp.jj[a];
      if (sj.ich != sj.jch) {
        if (qr == ii && qc == jj) {
          if (!touched) { val = *h; touched = true; }
          val = val + (sj.ich > sj.jch ? ysum(a, sj, lr + 1, lc + 1)
                                       : ysum(a, sj, lc + 1, lr + 1));
        }
      } else {
        if (qr == ii && qc == jj) {
          if (!touched) { val = *h; touched = true; }
          val = val + ysum(a, sj, lr + 1, lc + 1) / 2.0;
        }
        if (qr == jj && qc == ii) {
          if (!touched) { val = *h; touched = true; }
          val = val + ysum(a, sj, lc + 1, lr + 1) / 2.0;
        }
      }
    }
  }
  if (touched) *h = val;
}

}  // namespace

int ensure_fscratch(dbsrg_ctx *c, size_t bytes) {
  return grow_buffer(c, &c->fscratch, &c->fscratch_bytes, bytes);
}

// the four R^k vectors of one k over nb orbitals (b2o null: all of them)
static int r_far_vectors(dbsrg_ctx *c, int k, int nb, const int *b2o, double *W, float2 *Wf) {
  const DeviceGrid &g = c->g;
  const int ns = g.ns;
  const size_t m = (size_t)ns * nb;
  const CellData *pp, *qq;
  int rc;
  if ((rc = get_celldata(c, 0, 0, k, &pp)) || (rc = get_celldata(c, 0, 1, k, &qq)) ||
      (rc = moment_sums(c, 0, 0, k)))
    return rc;
  auto side = [&](int comp, const CellData &cd) {
    const int o = comp == 1 ? 0 : 2;
    return FarSide{1, 1, comp, cd.tlo1, cd.thi1, W + o * m, W + (o + 1) * m,
                   Wf ? Wf + o * m : nullptr, Wf ? Wf + (o + 1) * m : nullptr};
  };
  const dim3 gv((unsigned)((m + 63) / 64), 2);
  DBSRG_RUN(c, "k_far_vectors",
            k_far_vectors<<<gv, 64, 0, c->stream>>>(ns, g.ks, nb, b2o, c->pq, side(1, *pp),
                                                    side(2, *qq)));
  return DBSRG_OK;
}

int far_vectors_all(dbsrg_ctx *c, int k, double *W) {
  return r_far_vectors(c, k, c->nbf, nullptr, W, nullptr);
}

static int ensure_rfar(dbsrg_ctx *c, int k, RFar **out) {
  RFar &r = c->rfarw[k];
  if (!r.W) {
    const size_t m = (size_t)c->g.ns * c->nbound;
    CacheBuffer buf(c, 8 * m * sizeof(double));
    double *W = (double *)buf.p;
    if (!W) return set_err(c, DBSRG_ENOMEM, "far-field allocation failed");
    const int rc = r_far_vectors(c, k, c->nbound, c->b2o, W, (float2 *)(W + 4 * m));
    if (rc) return rc;
    buf.keep();
    r.W = W;
    r.Wf = (float2 *)(W + 4 * m);
  }
  *out = &r;
  return DBSRG_OK;
}

int get_rfar(dbsrg_ctx *c, int k, const double **W) {
  RFar *r;
  const int rc = ensure_rfar(c, k, &r);
  if (!rc) *W = r->W;
  return rc;
}

// far-field vectors of (family, type, k, exchange case), cached; R^k (case 3
// only): views of the four vectors that the types of the k share
static int get_farfield(dbsrg_ctx *c, int family, int type, int k, int cs, const FarField **out) {
  std::map<size_t, FarField> &v = family == 0 ? c->rfar : c->sfar;
  const size_t idx = ((size_t)k * (family == 0 ? 4 : 2) + type) * 2 + (cs == 4 ? 1 : 0);
  auto it = v.find(idx);
  if (it != v.end() && it->second.U) {
    *out = &it->second;
    return DBSRG_OK;
  }
  const DeviceGrid &g = c->g;
  const int ns = g.ns, nb = c->nbound;
  const size_t m = (size_t)ns * nb;
  const dim3 gv((unsigned)((m + 63) / 64), 2);
  const TableBases tb = table_bases(g, family, type);
  int rc;
  FarField f;
  if (family == 0) {
    if (cs != 3) return set_err(c, DBSRG_EINVAL, "far field: R^k exchange is convol case 3");
    RFar *rp;
    if ((rc = ensure_rfar(c, k, &rp))) return rc;
    RFar &r = *rp;
    // U, Ul: lo and hi of electron 1's pairs; V, Vl: hi and lo of electron 2's
    const int a = tb.a1 == 1 ? 0 : 2, b = tb.b1 == 1 ? 0 : 2;
    f.U = r.W + a * m;
    f.Ul = r.W + (a + 1) * m;
    f.V = r.W + (b + 1) * m;
    f.Vl = r.W + b * m;
    f.Vf = r.Wf + (b + 1) * m;
    f.Vlf = r.Wf + b * m;
    f.sh = &r;
    f.first = a;
  } else {
    const CellData *cd;
    if ((rc = get_celldata(c, family, type, k, &cd)) || (rc = moment_sums(c, family, type, k)))
      return rc;
    CacheBuffer buf(c, 3 * m * sizeof(double));
    double *base = (double *)buf.p;
    if (!base) return set_err(c, DBSRG_ENOMEM, "far-field allocation failed");
    f.U = base;
    f.V = base + m;
    f.Vf = (float2 *)(base + 2 * m);
    // electron 1: case 3 output = first function, contracted = second; electron 2:
    // output = second, contracted = first; case 4 the other way
    const int o1f = cs == 3 ? 1 : 0, o2f = 1 - o1f;
    const int cc1 = cs == 3 ? tb.a2 : tb.a1, cc2 = cs == 3 ? tb.b1 : tb.b2;
    const FarSide s1{0, o1f, cc1, cd->tlo1, nullptr, f.U, nullptr, nullptr, nullptr};
    const FarSide s2{0, o2f, cc2, cd->thi2, nullptr, f.V, nullptr, f.Vf, nullptr};
    DBSRG_RUN(c, "k_far_vectors",
              k_far_vectors<<<gv, 64, 0, c->stream>>>(ns, g.ks, nb, c->b2o, c->pq, s1, s2));
    buf.keep();
  }
  v[idx] = f;
  *out = &v.at(idx);
  return DBSRG_OK;
}

// bound-orbital rows of both components, built once per orbital set
static int ensure_brows(dbsrg_ctx *c) {
  if (c->brows) return DBSRG_OK;
  const int ns = c->g.ns, nb = c->nbound;
  const size_t m = (size_t)ns * nb;
  CacheBuffer buf(c, 4 * m * sizeof(double));
  double *rows = (double *)buf.p;
  if (!rows) return set_err(c, DBSRG_ENOMEM, "bound-orbital rows allocation failed");
  float2 *rowsf = (float2 *)(rows + 2 * m);
  DBSRG_RUN(c, "k_bound_rows",
            k_bound_rows<<<dim3((unsigned)((m + 255) / 256), 2), 256, 0, c->stream>>>(
                ns, nb, c->b2o, c->pq, rows, rowsf));
  buf.keep();
  c->brows = rows;
  c->browsf = rowsf;
  return DBSRG_OK;
}

int ensure_bound_rows(dbsrg_ctx *c, bool *built) {
  if (c->brows) return DBSRG_OK;
  *built = true;
  return ensure_brows(c);
}

static long long pairpot_key(int kind, int family, int type, int k, int icv, int jp1, int jp2,
                             bool ff) {
  return (long long)kind | (long long)family << 1 | (long long)type << 2 | (long long)icv << 5 |
         (long long)jp1 << 8 | (long long)jp2 << 10 | (long long)ff << 12 | (long long)k << 13;
}

static int set_smem(dbsrg_ctx *c, const void *fn, size_t smem) {
  if (smem > 220 * 1024) return set_err(c, DBSRG_EINVAL, "pair potentials: too many bound orbitals");
  return raise_smem_limit(c, fn, smem);
}

bool pair_potentials_fit(const dbsrg_ctx *c) {
  return c->g.ks <= FAR && c->nbound >= 1 && c->nbound <= 64;
}

// direct pair potentials of up to four tables of one family, cached: Kd[pair][ns*ncol]
// of (type, k, case icv) with density components jp1/jp2.  ff: the small
// matrices' contraction in float-float arithmetic and the results stored as
// float-float pairs (the split form's gather-sums read those).
int get_pairpots_direct(dbsrg_ctx *c, int n, const PairPotKey *want, bool ff, const void **out) {
  const DeviceGrid &g = c->g;
  const int ns = g.ns, ks = g.ks, nv = g.nv, kk = ks * ks, nb = c->nbound;
  const size_t npair = (size_t)nb * nb;
  int rc, m = 0, at[4];  // at: what builds want[i], -1 if cached
  long long keys[4];
  const PairPotKey *req[4];  // those to build
  for (int i = 0; i < n; i++) {
    const PairPotKey &w = want[i];
    const long long key = pairpot_key(0, w.family, w.type, w.k, w.icv, w.jp1, w.jp2, ff);
    auto it = c->ppot.find(key);
    at[i] = -1;
    if (it != c->ppot.end()) {
      out[i] = it->second;
      continue;
    }
    at[i] = (int)(std::find(keys, keys + m, key) - keys);
    if (at[i] < m) continue;  // wanted twice
    keys[m] = key;
    req[m++] = &w;
  }
  if (m == 0) return DBSRG_OK;
  if ((rc = ensure_brows(c))) return rc;
  const int family = req[0]->family;
  const char sym = family == 0 ? 's' : 'n';
  const int ncol = sym == 's' ? ks : 2 * ks - 1;
  const size_t per = (size_t)ns * ncol;
  const CellData *cd[4];
  TableBases tb[4];
  int np[4], symab[4], npmax = 0, k12 = 0;
  size_t sall = 0;  // scanned sums: SA, SB (nv x np) a table
  for (int i = 0; i < m; i++) {
    const PairPotKey &w = *req[i];
    if ((rc = get_celldata(c, family, w.type, w.k, &cd[i]))) return rc;
    tb[i] = table_bases(g, family, w.type);
    const PairSpec ed = w.icv == 1 ? tb[i].e2 : tb[i].e1;
    symab[i] = ed.sym && w.jp1 == w.jp2;
    np[i] = pair_count(nb, symab[i]);
    npmax = std::max(npmax, np[i]);
    k12 = std::max(k12, 3 * ed.k1 + ed.k2);
    sall += 2 * (size_t)np[i] * nv;
  }
  const int ps = c->stream == c->bstream[1] ? 1 : 0;  // scratch of this stream
  if (c->stream != c->bstream[0] && c->stream != c->bstream[1]) c->stream_built = true;
  if ((rc = ensure_pscratch(c, ps, sall * sizeof(double)))) return rc;
  double *K[4];  // doubles, or as many float2 pairs (same bytes)
  for (int i = 0; i < m; i++)
    if (!(K[i] = (double *)cache_alloc(c, npair * per * sizeof(double)))) {
      cudaGetLastError();
      while (i > 0) cache_free(c, K[--i]);
      return set_err(c, DBSRG_ENOMEM, "pair potential allocation failed");
    }
  cudaStream_t st = c->stream;
  PairCellArgs ca{};
  PairScanArgs sa{};
  double *S = (double *)c->pscratch[ps];
  for (int i = 0; i < m; i++) {
    const PairPotKey &w = *req[i];
    const bool one = w.icv == 1;
    ca.ed[i] = one ? tb[i].e2 : tb[i].e1;
    ca.symab[i] = symab[i];
    ca.M1[i] = one ? cd[i]->hi2 : cd[i]->lo1;
    ca.M2[i] = one && family == 0 ? cd[i]->lo2 : nullptr;
    ca.P1[i] = c->brows + (size_t)(w.jp1 - 1) * nb * ns;
    ca.P2[i] = c->brows + (size_t)(w.jp2 - 1) * nb * ns;
    ca.S1[i] = S;
    ca.S2[i] = ca.M2[i] ? S + (size_t)np[i] * nv : nullptr;
    S += 2 * (size_t)np[i] * nv;
    sa.np[i] = np[i];
    sa.suffix0[i] = one;
    sa.S[i][0] = ca.S1[i];
    sa.S[i][1] = ca.S2[i];
  }
  auto potentials = [&](auto ff_c, auto km_c) -> int {
    constexpr bool F = decltype(ff_c)::value;
    constexpr int KM = decltype(km_c)::value, PDW = pair_window(KM), PDR = pair_rows(KM);
    using T = typename Val<F>::T;
    const size_t sm1 = (size_t)nb * k12 * sizeof(double);
    PairDirArgs<F> d{};
    d.ns = ns;
    d.nv = nv;
    d.kk = kk;
    d.nb = nb;
    d.ncol = ncol;
    d.dl0 = sym == 's' ? 0 : 1 - ks;
    d.bw = (std::min(nb, PDB) + 1) & ~1;
    d.per = per;
    const T *rows = F ? (const T *)c->browsf : (const T *)c->brows;
    double fl = 0.0;
    for (int i = 0; i < m; i++) {
      const PairPotKey &w = *req[i];
      const bool one = w.icv == 1, ofirst = one != cd[i]->tr;
      PairDirTable<F> &t = d.t[i];
      t.np = np[i];
      t.symab = symab[i];
      t.suf = one;
      t.eo = one ? tb[i].e1 : tb[i].e2;
      t.ed = one ? tb[i].e2 : tb[i].e1;
      t.rkd = cd[i]->rkd;
      t.rcell = (size_t)npairs(t.eo) * npairs(t.ed);
      t.rpo = ofirst ? 1 : npairs(t.ed);
      t.rpd = ofirst ? npairs(t.eo) : 1;
      t.L1 = one ? cd[i]->lo1 : cd[i]->hi2;
      t.L2 = ca.M2[i] ? cd[i]->hi1 : nullptr;
      t.M1 = ca.M1[i];
      t.M2 = ca.M2[i];
      t.P1 = rows + (size_t)(w.jp1 - 1) * nb * ns;
      t.P2 = rows + (size_t)(w.jp2 - 1) * nb * ns;
      t.SA = ca.S1[i];
      t.SB = ca.S2[i];
      t.K = (T *)K[i];
      // executed work: an output's n = k - |dl| cells hold r = n + k - 1 functions
      // and a banded matrix of r^2 - n (n - 1) elements: as many multiply-adds per
      // second orbital, r + 2 per pair; the potentials written
      for (int col = 0; col < ncol; col++) {
        const int x = std::min(t.eo.k1, t.eo.k2) - std::abs(d.dl0 + col);
        if (x <= 0) continue;
        const double r = x + t.ed.k1 - 1;
        fl += 2.0 * ns * ((r * r - x * (x - 1.0)) * nb + (r + 2.0) * np[i]);
      }
    }
    const size_t smem = sizeof(T) * ((size_t)PDX * PDW * (PDW + d.bw) + PDR * d.bw +
                                     (size_t)PDR * pair_row_stride(nb));
    int frc = set_smem(c, (const void *)k_pair_cellsum, sm1);
    if (!frc) frc = set_smem(c, (const void *)k_pair_direct<F, KM>, smem);
    if (frc) return frc;
    DBSRG_RUN(c, "k_pair_cellsum",
              k_pair_cellsum<<<dim3(nv, m), 256, sm1, st>>>(ns, kk, nb, ca));
    DBSRG_RUN(c, "k_pair_scan",
              k_pair_scan<<<dim3((unsigned)((npmax + PSP - 1) / PSP), 2 * m), PSP * PSW, 0,
                               st>>>(nv, sa));
    const dim3 gd((unsigned)((ns + PDX - 1) / PDX), (unsigned)(ncol * m),
                  (unsigned)((nb + PDB - 1) / PDB));
    DBSRG_RUN_W(c, "k_pair_direct", 8.0 * (double)per * npair * m, fl,
                (k_pair_direct<F, KM><<<gd, PDT, smem, st>>>(d)));
    return DBSRG_OK;
  };
  const std::integral_constant<int, FAR> k9;
  const std::integral_constant<int, DBSRG_MAXK> kmax;
  if (ks <= FAR)
    rc = ff ? potentials(std::true_type(), k9) : potentials(std::false_type(), k9);
  else if (!ff)  // the energy functional; lists of the factored forms end at order 9
    rc = potentials(std::false_type(), kmax);
  else
    rc = set_err(c, DBSRG_EINVAL, "factored contraction: spline order above 9");
  for (int i = 0; i < m; i++) {
    if (rc)
      cache_free(c, K[i]);
    else
      c->ppot[keys[i]] = K[i];
  }
  if (rc) return rc;
  for (int i = 0; i < n; i++)
    if (at[i] >= 0) out[i] = K[at[i]];
  return DBSRG_OK;
}

// exchange band pair potentials of (family, type, k, case), cached:
// Kb[pair][ns*17], in FP64 or float-float pairs (ff: both stages in that
// arithmetic, same bytes; the split form's Z digits read those).  An R^k table's
// come with those of all types of its k (tabs of types 0..2 by type, type 3 from
// type 2), as a list takes them all; S^k: tabs[0].  The density components are
// the contracted functions' (factored_contract checks them).
static int get_pairpot_band(dbsrg_ctx *c, int family, int type, int k, int cs,
                            const double *const *tabs, bool ff, const void **out) {
  auto key_of = [&](int t) {
    const TableBases tb = table_bases(c->g, family, t);
    return pairpot_key(1, family, t, k, cs, cs == 3 ? tb.a2 : tb.a1, cs == 3 ? tb.b1 : tb.b2, ff);
  };
  auto it = c->ppot.find(key_of(type));
  if (it != c->ppot.end()) {
    *out = it->second;
    return DBSRG_OK;
  }
  const DeviceGrid &g = c->g;
  const int ns = g.ns, ks = g.ks, nb = c->nbound;
  const size_t npair = (size_t)nb * nb, per = (size_t)ns * NDB;
  int rc;
  if ((rc = ensure_brows(c))) return rc;
  const size_t kbytes = npair * per * sizeof(double);
  const int n = family == 0 ? 3 : 1;
  void *K[3], *Kx[3] = {nullptr, nullptr, nullptr};
  // the results, S^k one, R^k those of types 0..2 and of type 3 (type 2's with the
  // electrons exchanged)
  void *buf[4];
  for (int i = 0; i < n + (n == 3); i++)
    if (!(buf[i] = cache_alloc(c, kbytes))) {
      while (i > 0) cache_free(c, buf[--i]);
      return set_err(c, DBSRG_ENOMEM, "pair potential allocation failed");
    }
  for (int i = 0; i < n; i++) K[i] = buf[i];
  if (n == 3) Kx[0] = K[0], Kx[1] = K[1], Kx[2] = buf[3];
  const int W = 2 * ks - 1, mode = family == 0 ? 0 : (cs == 3 ? 1 : 2);
  const int bw = (std::min(nb, PDB) + 1) & ~1;
  auto potentials = [&](auto ff_c) -> int {
    constexpr bool F = decltype(ff_c)::value;
    using T = typename Val<F>::T;
    const T *rows = F ? (const T *)c->browsf : (const T *)c->brows;
    PairBandArgs<F> p{};
    p.ns = ns;
    p.ks = ks;
    p.nb = nb;
    p.mode = mode;
    p.bw = bw;
    for (int i = 0; i < n; i++) {
      const TableBases tb = table_bases(g, family, family == 0 ? i : type);
      p.rkb[i] = tabs[i];
      p.P1[i] = rows + (size_t)((cs == 3 ? tb.a2 : tb.a1) - 1) * nb * ns;
      p.P2[i] = rows + (size_t)((cs == 3 ? tb.b1 : tb.b2) - 1) * nb * ns;
      p.Kout[i] = (T *)K[i];
      p.Kx[i] = (T *)Kx[i];
      p.y0[i + 1] = p.y0[i] + (Kx[i] == K[i] ? BAND + 1 : NDB);
    }
    for (int i = n; i < 3; i++) p.y0[i + 1] = p.y0[i];
    const int ny = p.y0[n];
    if (n == 1) p.y0[1] = p.y0[2] = ny;
    const dim3 gb((unsigned)((ns + PXC - 1) / PXC), (unsigned)ny, (unsigned)((nb + PDB - 1) / PDB));
    // executed work: per output row and band diagonal W^2 nb (stage 1) and
    // W nb^2 (stage 2) multiply-adds; the band tables read, the potentials
    // written
    const double kb = family == 0 ? ks : W;
    const double bflops = 2.0 * ns * ny * ((double)W * W * nb + (double)W * nb * nb);
    const double bbytes = 8.0 * ns * NDB * (n * kb * kb + (n == 3 ? 4 : 1) * (double)npair);
    const size_t smem = sizeof(T) * ((size_t)PXC * PBW * (PBW + bw) + PBR * bw +
                                     (size_t)PBR * pair_row_stride(nb));
    const int brc = set_smem(c, (const void *)k_pair_band<F>, smem);
    if (brc) return brc;
    DBSRG_RUN_W(c, "k_pair_band", bbytes, bflops,
                k_pair_band<F><<<gb, PDT, smem, c->stream>>>(p));
    return DBSRG_OK;
  };
  rc = ff ? potentials(std::true_type()) : potentials(std::false_type());
  for (int i = 0; i < n + (n == 3); i++) {
    if (rc)
      cache_free(c, buf[i]);
    else
      c->ppot[key_of(n == 3 ? i : type)] = (double *)buf[i];
  }
  if (rc) return rc;
  *out = c->ppot.at(key_of(type));
  return DBSRG_OK;
}

std::set<const void *> orbital_products(const dbsrg_ctx *c) {
  std::set<const void *> v;
  for (const auto &kv : c->rfarw) v.insert({kv.second.W, kv.second.D});
  for (const auto &kv : c->sfar) v.insert({kv.second.U, kv.second.Ud});
  for (const auto &kv : c->ppot) v.insert(kv.second);
  for (const auto *q : {&c->quad, &c->quadb}) v.insert(q->begin(), q->end());
  v.insert({c->brows, c->vch});
  v.erase(nullptr);
  return v;
}

void drop_orbital_products(dbsrg_ctx *c, const std::set<const void *> &keep) {
  const std::set<const void *> all = orbital_products(c);
  if (std::includes(keep.begin(), keep.end(), all.begin(), all.end())) return;
  cudaStreamSynchronize(c->stream);
  auto kept = [&](const void *p) { return keep.count(p) != 0; };
  for (auto it = c->rfarw.begin(); it != c->rfarw.end();) {
    RFar &r = it->second;
    const bool w = kept(r.W), d = w && kept(r.D);
    // the types' views go with the vectors, their digits with the digits
    for (auto f = c->rfar.begin(); f != c->rfar.end();) {
      if (f->second.sh == &r && !d) f->second.Ud = nullptr, f->second.eu = nullptr;
      f = f->second.sh == &r && !w ? c->rfar.erase(f) : std::next(f);
    }
    if (!d) {
      cache_free(c, r.D);
      r.D = nullptr;
      r.e = nullptr;
    }
    if (!w) cache_free(c, r.W);
    it = w ? std::next(it) : c->rfarw.erase(it);
  }
  for (auto it = c->sfar.begin(); it != c->sfar.end();) {
    FarField &f = it->second;
    const bool u = kept(f.U);
    if (!u || !kept(f.Ud)) {
      cache_free(c, f.Ud);
      f.Ud = nullptr;
      f.eu = nullptr;
    }
    if (!u) cache_free(c, f.U);
    it = u ? std::next(it) : c->sfar.erase(it);
  }
  for (auto it = c->ppot.begin(); it != c->ppot.end();) {
    const bool k = kept(it->second);
    if (!k) cache_free(c, it->second);
    it = k ? std::next(it) : c->ppot.erase(it);
  }
  for (auto *q : {&c->quad, &c->quadb})
    for (double *&p : *q)
      if (!kept(p)) {
        cache_free(c, p);
        p = nullptr;
      }
  if (!kept(c->brows)) {
    cache_free(c, c->brows);
    c->brows = nullptr;
    c->browsf = nullptr;
  }
  if (!kept(c->vch)) {
    cache_free(c, c->vch);
    c->vch = nullptr;
  }
}

void free_orbital_products(dbsrg_ctx *c) {
  graph_drop(c);
  drop_orbital_products(c, {});
}

int factored_contract(dbsrg_ctx *c, const FactorJob &j) {
  const DeviceGrid &g = c->g;
  const int ns = g.ns, ks = g.ks, nb = c->nbound;
  cudaStream_t st = c->stream;
  int rc;
  if (nb < 1 || nb > NB_MAX)
    return set_err(c, DBSRG_EINVAL, "factored contraction: 1..128 bound orbitals (ipbs = 0)");
  if (ks > FAR) return set_err(c, DBSRG_EINVAL, "factored contraction: spline order above 9");
  if (j.nown < 1) return DBSRG_OK;
  QuadSpec qs{};
  qs.na = j.na;
  for (int a = 0; a < j.na; a++) {
    qs.ii[a] = j.ii[a];
    qs.jj[a] = j.jj[a];
  }
  if (j.icv >= 3 && j.split) {
    SplitExchange x{};
    x.na = j.na;
    x.nm = j.nm;
    x.lower = j.family == 0 ? 1 : 0;
    for (int a = 0; a < j.na; a++) {
      const int cs = j.icv;
      if ((rc = get_farfield(c, j.family, j.types[a], j.kpol, cs, &x.far[a]))) return rc;
      TableBases tb = table_bases(g, j.family, j.types[a]);
      int c1 = cs == 3 ? tb.a2 : tb.a1, c2 = cs == 3 ? tb.b1 : tb.b2;
      if (c1 != j.jp1[a] || c2 != j.jp2[a])
        return set_err(c, DBSRG_EINVAL, "factored exchange: component mismatch");
      if ((rc = get_pairpot_band(c, j.family, j.types[a], j.kpol, cs, j.tabs, true,
                                 (const void **)&x.Kbf[a])))
        return rc;
    }
    x.members = j.members;
    x.xq = j.xq;
    x.hxq = j.hxq;
    x.nxq = j.nxq;
    x.info = j.info;
    x.pairs = j.pairs;
    x.cd = j.cd;
    x.cdf = j.cdf;
    x.prep = j.prep;
    x.nent = j.nent;
    return split_exchange(c, x);
  }
  if (j.icv >= 3 && j.prep) {
    for (int a = 0; a < j.na; a++) {
      const FarField *f;
      const void *Kb;
      if ((rc = get_farfield(c, j.family, j.types[a], j.kpol, j.icv, &f))) return rc;
      if ((rc = get_pairpot_band(c, j.family, j.types[a], j.kpol, j.icv, j.tabs, false, &Kb)))
        return rc;
    }
    return DBSRG_OK;
  }
  if (j.icv >= 3) {
    const size_t per = (size_t)ns * ns;
    size_t zs = (size_t)j.nm * nb * ns;
    if ((rc = ensure_fscratch(c, 2 * zs * sizeof(double)))) return rc;
    double *Z = (double *)c->fscratch, *Zl = Z + zs;
    for (int a = 0; a < j.na; a++) {
      const int cs = j.icv;
      const FarField *f;
      if ((rc = get_farfield(c, j.family, j.types[a], j.kpol, cs, &f))) return rc;
      TableBases tb = table_bases(g, j.family, j.types[a]);
      int c1 = cs == 3 ? tb.a2 : tb.a1, c2 = cs == 3 ? tb.b1 : tb.b2;
      if (c1 != j.jp1[a] || c2 != j.jp2[a])
        return set_err(c, DBSRG_EINVAL, "factored exchange: component mismatch");
      const double *Kb;
      if ((rc = get_pairpot_band(c, j.family, j.types[a], j.kpol, cs, j.tabs, false,
                                 (const void **)&Kb)))
        return rc;
      double *Ya = j.Y + (size_t)a * j.nm * per;
      dim3 gz((unsigned)((ns * nb + 127) / 128), (unsigned)j.nm);
      DBSRG_RUN(c, "k_far_z",
                k_far_z<<<gz, 128, 0, st>>>(ns, nb, j.members, j.info, j.pairs, j.cd, f->V,
                                            f->Vl, Z, f->Vl ? Zl : nullptr));
      dim3 gf((unsigned)((ns + 31) / 32), (unsigned)((ns + 31) / 32), (unsigned)j.nm);
      DBSRG_RUN(c, "k_far_field",
                k_far_field<<<gf, 256, 0, st>>>(ns, nb, f->U, f->Ul, Z, f->Vl ? Zl : nullptr, Ya,
                                                per));
      dim3 gb((unsigned)((ns * NDB + 255) / 256), (unsigned)j.nm);
      DBSRG_RUN(c, "k_band_sum",
                k_band_sum<<<gb, 256, 0, st>>>(ns, j.members, j.info, j.pairs, j.cd, Kb, Ya, per));
    }
    const int nt = (ns + 31) / 32;
    dim3 gs((unsigned)(4 * nt * nt), (unsigned)j.nown);
    DBSRG_RUN(c, "k_scatter_x",
              k_scatter_x<<<gs, 256, 0, st>>>(ns, qs, j.nm, j.members, j.own, j.info, j.Y,
                                              j.family == 0 ? 1 : 0, hch_base(c)));
    return DBSRG_OK;
  }
  if (j.dseg) return direct_segments(c, j);
  // direct, from the pair potentials
  KdSet kd{};
  const bool ff = j.split && j.cdf;
  PairPotKey want[4];
  const void *got[4];
  for (int a = 0; a < j.na; a++)
    want[a] = {j.family, j.types[a], j.kpol, j.icv, j.jp1[a], j.jp2[a]};
  if ((rc = get_pairpots_direct(c, j.na, want, ff, got))) return rc;
  for (int a = 0; a < j.na; a++) {
    if (ff)
      kd.Kf[a] = (const float2 *)got[a];
    else
      kd.K[a] = (const double *)got[a];
  }
  if (j.prep) return DBSRG_OK;
  const size_t space = (size_t)4 * ns * (2 * ks - 1);
  dim3 gs((unsigned)((space + 127) / 128), (unsigned)j.nown);
  // executed work: per PQ type every band element of its quadrant (about
  // ns (2ks-1)) sums one pair-potential value per entry of the owner and
  // partner segments (one multiply-add, float-float in the split form), and
  // is read and written once in hch; the potentials are read per entry
  const double nd = 2.0 * ks - 1.0, band = ns * nd;
  const double wflops = 2.0 * j.na * band * (double)j.nent;
  const double wbytes = 16.0 * j.na * band * j.nown + 8.0 * j.na * band * (double)j.nent;
  if (j.split && j.cdf)
    DBSRG_RUN_W(c, "k_scatter_dp", wbytes, wflops,
                k_scatter_dp<true><<<gs, 128, 0, st>>>(ns, ks, j.sym, qs, kd, j.members, j.own,
                                                       j.info, j.pairs, j.cd, j.cdf, hch_base(c)));
  else
    DBSRG_RUN_W(c, "k_scatter_dp", wbytes, wflops,
                k_scatter_dp<false><<<gs, 128, 0, st>>>(ns, ks, j.sym, qs, kd, j.members, j.own,
                                                        j.info, j.pairs, j.cd, j.cdf,
                                                        hch_base(c)));
  return DBSRG_OK;
}
