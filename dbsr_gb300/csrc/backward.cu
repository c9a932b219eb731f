// backward.cu -- the energy functional E = sum_e c_e R^k_e(a,b;c,d) over the
// bound orbitals and its gradient with respect to their P/Q B-spline
// coefficients (the direct potentials DBSR_HF and DBSR_MCHF build in their
// SCF step, hf_matrix.f90:2-163).
//
// R^k(a,b;c,d) (rk, dbsr_lib_dbs.f90:3981-4022) sums four table types t with
// electron-1 basis A_t and electron-2 basis B_t (0 PP|PP, 1 QQ|QQ,
// 2 PP|QQ, 3 QQ|PP): R_t = rho1^T T_t rho2 with rho1 the symmetric band
// density of (a,c) in basis A_t and rho2 that of (b,d) in basis B_t.  The
// direct pair potential Kd_t[(b,d)] (factor.cu; the convol case 1 of T_t
// with rho2) is the potential rho2 makes for electron 1.  The tables are
// symmetric under exchanging the electrons with types 2 and 3 swapped, so
// with
//   V_P[(p,q)] = Kd_0[(p,q)] + Kd_2[(p,q)],  V_Q = Kd_1 + Kd_3,
// the potential that the whole density of the pair makes for a P or a Q
// function of the other electron (symmetric band matrices, the same for
// (q,p)), an entry c R^k(a,b;c,d) adds c V_X[(b,d)] to the potential W_X of
// the pair {a,c} and c V_X[(a,c)] to that of {b,d}, and
//   dE/df_u += W_X{u,v} f_v,  dE/df_v += W_X{u,v} f_u  (component X),
//   E = 1/2 sum over {u,v}, X of f_u W_X{u,v} f_v
// (without the gradient, only the first of the two and E without the 1/2).
// So the work is one sum of band potentials per (k, pair), in entry order
// from a host-built list, and two band products; the terms are summed per
// (orbital, component) in a fixed order: deterministic, no atomics.
// The pair potentials are built from the cell moments and diagonal cells,
// recomputed when the tables were released.
#include "internal.cuh"

#include <algorithm>

namespace {

struct KdTypes {
  const double *K[4];  // Kd_t[pair][ns*ks], 's' storage
};

// V[X][up][q] = Kd_t0[pair][q] + Kd_t1[pair][q] over the unordered bound pairs
// (upair: their ordered index), X = P: t = 0, 2; X = Q: t = 1, 3
__global__ void k_rk_vsum(size_t per, int nup, const int *upair, KdTypes kd, double *V) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= per) return;
  const int up = blockIdx.y, X = blockIdx.z;
  const size_t o = (size_t)upair[up] * per + q;
  V[((size_t)X * nup + up) * per + q] = kd.K[X][o] + kd.K[X + 2][o];
}

// One item = one (multipole, unordered pair {u,v}) with its list of (pair,
// coefficient); a block takes MC rows m of one component X of an item.  It
// forms the rows of W_X that those rows meet (ks - 1 before them as well) in
// shared memory, one thread per band element, the potentials of UE entries
// loaded together; then row m of W f_v and of W f_u (128 threads each).
// Bound by the L2 reads of the potentials: 16 ks bytes per row, entry and
// component.  ns 300, 30 orbitals, 5e4 entries of k = 0..8: 1e5 list
// positions.  One thread per (entry, type, role, row) with 17-term sums and a
// launch per run of entries took 355 ms of the evaluation's 367.7 (44 453
// launches, and the terms of every entry written and read back); with this
// kernel the evaluation takes 5.3 ms, 2.7 of them the pair potentials.
constexpr int MC = 128;
constexpr int UE = 4;
__global__ void __launch_bounds__(2 * MC) k_rk_pot(int ns, int ks, int nup, size_t per,
                                                   const int *istart, const int2 *iuv,
                                                   const int *lpair, const double *lcoef,
                                                   const double *V, const double *pq, int grad,
                                                   double *T, double *Epart) {
  extern __shared__ double W[];  // [ks][MC + ks - 1]
  __shared__ double wsum[MC / 32];
  const int m0 = blockIdx.x * MC, it = blockIdx.y, X = blockIdx.z;
  const int nr = MC + ks - 1, r0 = m0 - (ks - 1);
  const int e0 = istart[it], e1 = istart[it + 1];
  const double *Vx = V + (size_t)X * nup * per;
  for (int el = threadIdx.x; el < nr * ks; el += 2 * MC) {
    const int i = r0 + el % nr, dl = el / nr;
    double acc = 0.0;
    if (i >= 0 && i + dl < ns) {
      const double *v = Vx + (size_t)i + (size_t)ns * dl;
      int e = e0;
      for (; e + UE <= e1; e += UE) {
        double k[UE];
#pragma unroll
        for (int u = 0; u < UE; u++) k[u] = v[(size_t)lpair[e + u] * per];
#pragma unroll
        for (int u = 0; u < UE; u++) acc = fma(lcoef[e + u], k[u], acc);
      }
      for (; e < e1; e++) acc = fma(lcoef[e], v[(size_t)lpair[e] * per], acc);
    }
    W[el] = acc;
  }
  __syncthreads();
  const int role = threadIdx.x / MC, ml = threadIdx.x % MC, m = m0 + ml;
  const int2 uv = iuv[it];
  const double *fu = pq + (size_t)2 * ns * (uv.x - 1) + (size_t)ns * X;
  const double *fv = pq + (size_t)2 * ns * (uv.y - 1) + (size_t)ns * X;
  const double *f = role == 0 ? fv : fu;
  double acc = 0.0;
  if (m < ns && (grad || role == 0)) {
    for (int j = max(0, m - ks + 1); j <= min(ns - 1, m + ks - 1); j++) {
      const int lo = min(m, j), dl = abs(m - j);
      acc = fma(W[(lo - r0) + nr * dl], f[j], acc);
    }
    if (grad) T[(((size_t)it * 2 + X) * 2 + role) * ns + m] = acc;
  }
  if (role == 0) {
    double s = m < ns ? fu[m] * acc : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (ml % 32 == 0) wsum[ml / 32] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < MC / 32; w++) s += wsum[w];
    Epart[((size_t)it * 2 + X) * gridDim.x + blockIdx.x] = s;
  }
}

// E = f sum of n partial energies in a fixed order (one block, fixed tree)
__global__ void k_energy_sum(int n, double f, const double *R, double *E) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int e = threadIdx.x; e < n; e += 256) s += R[e];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *E = f * sh[0];
}

// grad[(o, comp, m)] = the terms of orbital o (lidx: 2 item + role) in a fixed
// order: GS slices of the list summed side by side, then the slices in order
constexpr int GS = 8;
__global__ void __launch_bounds__(32 * GS) k_rk_grad_reduce(int ns, const int *lstart,
                                                            const int *lidx, const double *T,
                                                            double *grad) {
  __shared__ double sh[GS][32];
  const int tx = threadIdx.x % 32, sl = threadIdx.x / 32;
  const int m = blockIdx.x * 32 + tx, o = blockIdx.y, X = blockIdx.z;
  double acc = 0.0;
  if (m < ns)
    for (int l = lstart[o] + sl; l < lstart[o + 1]; l += GS) {
      const int r = lidx[l];
      acc += T[(((size_t)(r >> 1) * 2 + X) * 2 + (r & 1)) * ns + m];
    }
  sh[sl][tx] = acc;
  __syncthreads();
  if (sl == 0 && m < ns) {
    for (int k = 1; k < GS; k++) acc += sh[k][tx];
    grad[((size_t)o * 2 + X) * ns + m] = acc;  // pq layout
  }
}

}  // namespace

extern "C" int dbsrg_backward(dbsrg_ctx *c, int n, const int *k, const int *i1, const int *i2,
                              const int *i3, const int *i4, const double *coef, double *energy,
                              double *grad) {
  if (!c) return DBSRG_EINVAL;
  int rc;
  if (n < 0 || (n > 0 && (!k || !i1 || !i2 || !i3 || !i4 || !coef)) || !energy)
    return set_err(c, DBSRG_EINVAL, "backward: bad arguments");
  if (!c->pq) return set_err(c, DBSRG_ESTATE, "backward: no orbitals set");
  cudaSetDevice(c->device);
  if (c->pending && (rc = drain(c))) return rc;
  const int ns = c->g.ns, ks = c->g.ks, nbf = c->nbf, nb = c->nbound;
  cudaStream_t st = c->stream;
  // the entries on the host (small: integer keys and coefficients)
  std::vector<int> hk(n), h1(n), h2(n), h3(n), h4(n);
  std::vector<double> hc(n);
  auto fetch = [&](void *dst, const void *src, size_t bytes) -> int {
    if (!bytes) return DBSRG_OK;
    DBSRG_TRY(c, cudaMemcpy(dst, src, bytes,
                            is_device_ptr(src) ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost));
    return DBSRG_OK;
  };
  const size_t ib = sizeof(int) * (size_t)n;
  if ((rc = fetch(hk.data(), k, ib)) || (rc = fetch(h1.data(), i1, ib)) ||
      (rc = fetch(h2.data(), i2, ib)) || (rc = fetch(h3.data(), i3, ib)) ||
      (rc = fetch(h4.data(), i4, ib)) || (rc = fetch(hc.data(), coef, sizeof(double) * n)))
    return rc;
  for (int e = 0; e < n; e++) {
    for (int o : {h1[e], h2[e], h3[e], h4[e]})
      if (o < 1 || o > nbf || c->h_bmap[o - 1] < 0)
        return set_err(c, DBSRG_EINVAL, "backward: orbitals must be bound orbitals 1..nbf");
    if (hk[e] < 0 || hk[e] > 63) return set_err(c, DBSRG_ERANGE, "backward: k out of range");
  }
  if (nb < 1 || nb > 64)
    return set_err(c, DBSRG_EINVAL, "backward: 1..64 bound orbitals (ipbs = 0)");
  // items: (multipole, unordered bound pair), each with the pairs and
  // coefficients of its list in entry order (counting sort)
  const bool want_grad = grad != nullptr;
  auto upair = [&](int o1, int o2) {
    const int x = c->h_bmap[o1 - 1], y = c->h_bmap[o2 - 1], lo = std::min(x, y), hi = std::max(x, y);
    return hi * (hi + 1) / 2 + lo;
  };
  const int nup = nb * (nb + 1) / 2;
  std::vector<int> up(nup), p1(n), p2(n);
  for (int hi = 0; hi < nb; hi++)
    for (int lo = 0; lo <= hi; lo++) up[hi * (hi + 1) / 2 + lo] = lo * nb + hi;
  int kmax = -1;
  for (int e = 0; e < n; e++) {
    p1[e] = upair(h1[e], h3[e]);
    p2[e] = upair(h2[e], h4[e]);
    kmax = std::max(kmax, hk[e]);
  }
  std::vector<int> pos((size_t)(kmax + 1) * nup + 1, 0);
  for (int e = 0; e < n; e++) {
    pos[(size_t)hk[e] * nup + p1[e] + 1]++;
    if (want_grad) pos[(size_t)hk[e] * nup + p2[e] + 1]++;
  }
  std::vector<int> istart, kitem(kmax + 2, 0);  // list start of each item; first item of each k
  std::vector<int2> iuv;
  std::vector<int> b2o(nb);
  for (int o = 0; o < nbf; o++)
    if (c->h_bmap[o] >= 0) b2o[c->h_bmap[o]] = o + 1;
  for (int k1 = 0; k1 <= kmax; k1++) {
    kitem[k1] = (int)iuv.size();
    for (int u = 0; u < nup; u++) {
      const size_t q = (size_t)k1 * nup + u;
      if (pos[q + 1]) {
        istart.push_back(pos[q]);
        iuv.push_back(make_int2(b2o[up[u] / nb], b2o[up[u] % nb]));
      }
      pos[q + 1] += pos[q];
    }
  }
  const int nitem = (int)iuv.size(), nl = kmax < 0 ? 0 : pos.back();
  if (kmax >= 0) kitem[kmax + 1] = nitem;
  istart.push_back(nl);
  std::vector<int> lpair(nl);
  std::vector<double> lcoef(nl);
  for (int e = 0; e < n; e++) {
    const size_t q = (size_t)hk[e] * nup;
    int &x = pos[q + p1[e]];
    lpair[x] = p2[e];
    lcoef[x++] = hc[e];
    if (want_grad) {
      int &y = pos[q + p2[e]];
      lpair[y] = p1[e];
      lcoef[y++] = hc[e];
    }
  }
  // gradient terms of every orbital: 2 item + role (0: target u, 1: target v)
  std::vector<int> lstart((size_t)nbf + 1, 0), lidx;
  if (want_grad) {
    for (const int2 &x : iuv) {
      lstart[x.x]++;
      lstart[x.y]++;
    }
    for (int o = 0; o < nbf; o++) lstart[o + 1] += lstart[o];
    lidx.resize((size_t)2 * nitem);
    std::vector<int> fill(lstart.begin(), lstart.end() - 1);
    for (int i = 0; i < nitem; i++) {
      lidx[fill[iuv[i].x - 1]++] = 2 * i;
      lidx[fill[iuv[i].y - 1]++] = 2 * i + 1;
    }
  }
  const size_t per = (size_t)ns * ks, ng = (size_t)ns * 2 * nbf;
  const int nmc = (ns + MC - 1) / MC;
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t tn = want_grad ? (size_t)nitem * 4 * ns : 0, vn = 2 * (size_t)nup * per;
  const size_t en = (size_t)nitem * 2 * nmc;
  const size_t bytes = al(4 * (size_t)nup) + al(4 * istart.size()) + al(8 * (size_t)nitem) +
                       al(4 * (size_t)nl) + al(8 * (size_t)nl) + al(8 * vn) + al(8 * tn) +
                       al(8 * en) + al(4 * lstart.size()) + al(4 * lidx.size()) + al(8 * ng) + 512;
  if ((rc = ensure_scratch(c, bytes))) return rc;
  char *base = (char *)c->scratch;
  auto take = [&](size_t b) {
    char *p = base;
    base += al(b);
    return (void *)p;
  };
  int *dup = (int *)take(4 * (size_t)nup), *dis = (int *)take(4 * istart.size());
  int2 *duv = (int2 *)take(8 * (size_t)nitem);
  int *dlp = (int *)take(4 * (size_t)nl);
  double *dlc = (double *)take(8 * (size_t)nl), *dV = (double *)take(8 * vn);
  double *dT = (double *)take(8 * tn), *dEp = (double *)take(8 * en);
  int *dls = (int *)take(4 * lstart.size()), *dli = (int *)take(4 * lidx.size());
  double *dG = (double *)take(8 * ng);
  double *dE = (double *)take(sizeof(double));
  if ((rc = copy_in(c, dup, up.data(), 4 * (size_t)nup)) ||
      (rc = copy_in(c, dis, istart.data(), 4 * istart.size())) ||
      (rc = copy_in(c, duv, iuv.data(), 8 * (size_t)nitem)) ||
      (rc = copy_in(c, dlp, lpair.data(), 4 * (size_t)nl)) ||
      (rc = copy_in(c, dlc, lcoef.data(), 8 * (size_t)nl)))
    return rc;
  if (want_grad && ((rc = copy_in(c, dls, lstart.data(), 4 * lstart.size())) ||
                    (rc = copy_in(c, dli, lidx.data(), 4 * lidx.size()))))
    return rc;
  // per multipole: the four pair potentials, their sums, the items
  const size_t smem = (size_t)(MC + ks - 1) * ks * sizeof(double);
  for (int kp = 0; kp <= kmax; kp++) {
    const int i0 = kitem[kp], ni = kitem[kp + 1] - i0;
    if (ni == 0) continue;
    KdTypes kd{};
    PairPotKey want[4];
    for (int t = 0; t < 4; t++) {
      const int comp = (t == 0 || t == 3) ? 1 : 2;  // electron-2 basis of the table
      want[t] = {0, t, kp, 1, comp, comp};
    }
    if ((rc = get_pairpots_direct(c, 4, want, false, (const void **)kd.K))) return rc;
    DBSRG_RUN(c, "k_rk_vsum",
              k_rk_vsum<<<dim3((unsigned)((per + 255) / 256), (unsigned)nup, 2), 256, 0, st>>>(
                  per, nup, dup, kd, dV));
    DBSRG_RUN(c, "k_rk_pot",
              k_rk_pot<<<dim3((unsigned)nmc, (unsigned)ni, 2), 2 * MC, smem, st>>>(
                  ns, ks, nup, per, dis + i0, duv + i0, dlp, dlc, dV, c->pq, want_grad ? 1 : 0,
                  dT + (want_grad ? (size_t)i0 * 4 * ns : 0), dEp + (size_t)i0 * 2 * nmc));
  }
  if (n > 0)
    DBSRG_RUN(c, "k_energy_sum",
              k_energy_sum<<<1, 256, 0, st>>>((int)en, want_grad ? 0.5 : 1.0, dEp, dE));
  else DBSRG_TRY(c, cudaMemsetAsync(dE, 0, sizeof(double), st));
  if (want_grad) {
    DBSRG_RUN(c, "k_rk_grad_reduce",
              k_rk_grad_reduce<<<dim3((unsigned)((ns + 31) / 32), (unsigned)nbf, 2), 32 * GS, 0,
                                 st>>>(ns, dls, dli, dT, dG));
    if ((rc = copy_out(c, grad, dG, sizeof(double) * ng))) return rc;
  }
  return copy_out(c, energy, dE, sizeof(double));
}
