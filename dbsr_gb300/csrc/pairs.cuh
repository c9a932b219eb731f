// pairs.cuh -- the pair numbering of cell moments and diagonal-cell integrals
// and the bases of a table's four functions, shared by the factored
// contractions (factor.cu, direct.cu).
#pragma once
#include "internal.cuh"

struct PairSpec {
  int k1, k2, sym;  // orders of the first / second function; packed symmetric
};

__device__ __forceinline__ int pidx(PairSpec s, int h1, int h2) {  // 1-based locals
  if (s.sym) {
    int a = min(h1, h2), b = max(h1, h2);
    return (a - 1) * s.k1 - ((a - 1) * (a - 2)) / 2 + (b - a);
  }
  return (h1 - 1) * s.k2 + (h2 - 1);
}
__host__ __device__ inline int npairs(PairSpec s) { return s.sym ? s.k1 * (s.k1 + 1) / 2 : s.k1 * s.k2; }

// bases of the four functions of a table: 1 = P, 2 = Q
struct TableBases {
  int a1, a2, b1, b2;
  PairSpec e1, e2;
};

inline TableBases table_bases(const DeviceGrid &g, int family, int type) {
  TableBases t;
  auto ord = [&](int b) { return b == 1 ? g.ksp : g.ksq; };
  if (family == 0) {
    int A = (type == 0 || type == 2) ? 1 : 2, B = (type == 0 || type == 3) ? 1 : 2;
    t.a1 = t.a2 = A;
    t.b1 = t.b2 = B;
    t.e1 = {ord(A), ord(A), 1};
    t.e2 = {ord(B), ord(B), 1};
  } else {
    t.a1 = 1;
    t.a2 = 2;
    t.b1 = type == 0 ? 1 : 2;
    t.b2 = type == 0 ? 2 : 1;
    t.e1 = {g.ksp, g.ksq, 0};
    t.e2 = {ord(t.b1), ord(t.b2), 0};
  }
  return t;
}
