// Generated by nrg_b200/gen_mech.py from KONNOV.txt: do not edit.
// Straight-line right-hand side and analytic iteration matrix over the
// 13 reacting species and 67 distinct reactions, and the right-hand side
// over all 13 species and 71 reactions; same operation order as the
// table-driven loops in chem_bdf.cuh, with the same explicitly rounded
// (never fused) operations.
#pragma once

namespace nrg {
namespace gen_konnov {

constexpr int kSpecN = 13, kSpecR = 67;
constexpr int kSpecLeft[67][3] = {
    {4, 4, -1},
    {4, 4, 0},
    {4, 4, 2},
    {4, 4, 4},
    {3, 3, -1},
    {3, 4, -1},
    {6, -1, -1},
    {6, 6, -1},
    {4, 1, -1},
    {8, -1, -1},
    {3, 0, -1},
    {4, 1, -1},
    {0, 5, -1},
    {5, 5, -1},
    {7, 3, -1},
    {4, 7, -1},
    {6, 3, -1},
    {0, 1, -1},
    {7, 5, -1},
    {7, 7, -1},
    {8, 4, -1},
    {8, 4, -1},
    {8, 3, -1},
    {8, 5, -1},
    {1, 3, -1},
    {12, 3, -1},
    {12, 3, -1},
    {3, 3, -1},
    {11, -1, -1},
    {11, 3, -1},
    {11, 4, -1},
    {11, 3, -1},
    {11, 12, -1},
    {9, 11, -1},
    {9, 1, -1},
    {9, 1, -1},
    {9, -1, -1},
    {9, 2, -1},
    {9, 12, -1},
    {9, 12, -1},
    {0, 11, -1},
    {4, 11, -1},
    {4, 11, -1},
    {7, 5, -1},
    {5, 11, -1},
    {12, 4, -1},
    {12, 5, -1},
    {12, 7, -1},
    {4, 7, -1},
    {9, 0, -1},
    {9, 6, -1},
    {3, 4, -1},
    {10, 1, -1},
    {10, 2, -1},
    {10, 6, -1},
    {10, 0, -1},
    {10, 5, -1},
    {10, 4, -1},
    {10, 3, -1},
    {10, 0, -1},
    {10, 1, -1},
    {10, 1, -1},
    {10, 6, -1},
    {4, 1, 4},
    {4, 1, 4},
    {4, 1, 3},
    {4, 1, 5},
};
constexpr int kSpecRight[67][3] = {
    {0, -1, -1},
    {0, 0, -1},
    {0, 2, -1},
    {0, 4, -1},
    {1, -1, -1},
    {5, -1, -1},
    {4, 5, -1},
    {4, 5, 6},
    {7, -1, -1},
    {5, 5, -1},
    {5, 4, -1},
    {5, 3, -1},
    {6, 4, -1},
    {6, 3, -1},
    {5, 1, -1},
    {5, 5, -1},
    {4, 7, -1},
    {4, 7, -1},
    {6, 1, -1},
    {8, 1, -1},
    {7, 0, -1},
    {6, 5, -1},
    {7, 5, -1},
    {7, 6, -1},
    {12, -1, -1},
    {1, 1, -1},
    {11, 1, -1},
    {11, -1, -1},
    {1, -1, -1},
    {1, 3, -1},
    {1, 4, -1},
    {3, 1, -1},
    {1, 1, 3},
    {3, 1, -1},
    {3, 11, -1},
    {3, 1, -1},
    {3, -1, -1},
    {3, 2, -1},
    {1, 3, 3},
    {1, 1, -1},
    {4, 7, -1},
    {5, 3, -1},
    {7, -1, -1},
    {6, 11, -1},
    {3, 7, -1},
    {5, 1, -1},
    {7, 1, -1},
    {5, 1, 1},
    {6, 9, -1},
    {5, 4, -1},
    {5, 5, -1},
    {10, -1, -1},
    {5, 1, -1},
    {5, 2, -1},
    {5, 6, -1},
    {5, 0, -1},
    {5, 5, -1},
    {5, 4, -1},
    {5, 3, -1},
    {6, 4, -1},
    {12, 4, -1},
    {7, 3, -1},
    {8, 4, -1},
    {0, 1, -1},
    {5, 5, -1},
    {5, 1, -1},
    {6, 1, -1},
};
constexpr int kSpecNupd[67] = {3, 5, 5, 5, 3, 3, 3, 5, 3, 3, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 3, 4, 4, 3, 2, 4, 4, 4, 5, 4, 4, 4, 2, 4, 5, 4, 4, 4, 3, 4, 4, 4, 4, 5, 4, 4, 4, 3, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 5, 5, 5, 5};
constexpr int kSpecUpdK[67][6] = {
    {0, 4, 4, 0, 0, 0},
    {0, 0, 0, 4, 4, 0},
    {0, 2, 2, 4, 4, 0},
    {0, 4, 4, 4, 4, 0},
    {1, 3, 3, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {4, 5, 6, 0, 0, 0},
    {4, 5, 6, 6, 6, 0},
    {1, 4, 7, 0, 0, 0},
    {5, 5, 8, 0, 0, 0},
    {0, 3, 4, 5, 0, 0},
    {1, 3, 4, 5, 0, 0},
    {0, 4, 5, 6, 0, 0},
    {3, 5, 5, 6, 0, 0},
    {1, 3, 5, 7, 0, 0},
    {4, 5, 5, 7, 0, 0},
    {3, 4, 6, 7, 0, 0},
    {0, 1, 4, 7, 0, 0},
    {1, 5, 6, 7, 0, 0},
    {1, 7, 7, 8, 0, 0},
    {0, 4, 7, 8, 0, 0},
    {4, 5, 6, 8, 0, 0},
    {3, 5, 7, 8, 0, 0},
    {5, 6, 7, 8, 0, 0},
    {1, 3, 12, 0, 0, 0},
    {1, 1, 3, 12, 0, 0},
    {1, 3, 11, 12, 0, 0},
    {3, 3, 11, 0, 0, 0},
    {1, 11, 0, 0, 0, 0},
    {1, 3, 3, 11, 0, 0},
    {1, 4, 4, 11, 0, 0},
    {1, 3, 3, 11, 0, 0},
    {1, 1, 3, 11, 12, 0},
    {1, 3, 9, 11, 0, 0},
    {1, 3, 9, 11, 0, 0},
    {1, 1, 3, 9, 0, 0},
    {3, 9, 0, 0, 0, 0},
    {2, 2, 3, 9, 0, 0},
    {1, 3, 3, 9, 12, 0},
    {1, 1, 9, 12, 0, 0},
    {0, 4, 7, 11, 0, 0},
    {3, 4, 5, 11, 0, 0},
    {4, 7, 11, 0, 0, 0},
    {5, 6, 7, 11, 0, 0},
    {3, 5, 7, 11, 0, 0},
    {1, 4, 5, 12, 0, 0},
    {1, 5, 7, 12, 0, 0},
    {1, 1, 5, 7, 12, 0},
    {4, 6, 7, 9, 0, 0},
    {0, 4, 5, 9, 0, 0},
    {5, 5, 6, 9, 0, 0},
    {3, 4, 10, 0, 0, 0},
    {1, 1, 5, 10, 0, 0},
    {2, 2, 5, 10, 0, 0},
    {5, 6, 6, 10, 0, 0},
    {0, 0, 5, 10, 0, 0},
    {5, 5, 5, 10, 0, 0},
    {4, 4, 5, 10, 0, 0},
    {3, 3, 5, 10, 0, 0},
    {0, 4, 6, 10, 0, 0},
    {1, 4, 10, 12, 0, 0},
    {1, 3, 7, 10, 0, 0},
    {4, 6, 8, 10, 0, 0},
    {0, 1, 1, 4, 4, 0},
    {1, 4, 4, 5, 5, 0},
    {1, 1, 3, 4, 5, 0},
    {1, 1, 4, 5, 6, 0},
};
constexpr int kSpecUpdProd[67][6] = {
    {1, 0, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 0, 0, 1, 0},
    {1, 0, 0, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 1, 0, 0, 1, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 0, 0, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 1, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 1, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 0, 1, 1, 0},
    {0, 1, 0, 0, 1, 0},
    {0, 1, 0, 0, 1, 0},
};

// zd = dC/dt at z (shared scratch in, shared scratch out)
template <class S>
__device__ __forceinline__ void spec_rhs(S& c) {
  const double z0 = c.z(0);
  const double z1 = c.z(1);
  const double z2 = c.z(2);
  const double z3 = c.z(3);
  const double z4 = c.z(4);
  const double z5 = c.z(5);
  const double z6 = c.z(6);
  const double z7 = c.z(7);
  const double z8 = c.z(8);
  const double z9 = c.z(9);
  const double z10 = c.z(10);
  const double z11 = c.z(11);
  const double z12 = c.z(12);
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0, d9 = 0.0, d10 = 0.0, d11 = 0.0, d12 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z4), z4);
  b = __dmul_rn(c.kr(0), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(1), z4), z4), z0);
  b = __dmul_rn(__dmul_rn(c.kr(1), z0), z0);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(2), z4), z4), z2);
  b = __dmul_rn(__dmul_rn(c.kr(2), z0), z2);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(3), z4), z4), z4);
  b = __dmul_rn(__dmul_rn(c.kr(3), z0), z4);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(4), z3), z3);
  b = __dmul_rn(c.kr(4), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z3), z4);
  b = __dmul_rn(c.kr(5), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(c.kf(6), z6);
  b = __dmul_rn(__dmul_rn(c.kr(6), z4), z5);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(7), z6), z6);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(7), z4), z5), z6);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z4), z1);
  b = __dmul_rn(c.kr(8), z7);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(c.kf(9), z8);
  b = __dmul_rn(__dmul_rn(c.kr(9), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(10), z3), z0);
  b = __dmul_rn(__dmul_rn(c.kr(10), z5), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z4), z1);
  b = __dmul_rn(__dmul_rn(c.kr(11), z5), z3);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(12), z0), z5);
  b = __dmul_rn(__dmul_rn(c.kr(12), z6), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(13), z5), z5);
  b = __dmul_rn(__dmul_rn(c.kr(13), z6), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(14), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(14), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z4), z7);
  b = __dmul_rn(__dmul_rn(c.kr(15), z5), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z6), z3);
  b = __dmul_rn(__dmul_rn(c.kr(16), z4), z7);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z0), z1);
  b = __dmul_rn(__dmul_rn(c.kr(17), z4), z7);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(18), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(19), z7), z7);
  b = __dmul_rn(__dmul_rn(c.kr(19), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(20), z7), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(21), z6), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(22), z8), z3);
  b = __dmul_rn(__dmul_rn(c.kr(22), z7), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z8), z5);
  b = __dmul_rn(__dmul_rn(c.kr(23), z7), z6);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(24), z1), z3);
  b = __dmul_rn(c.kr(24), z12);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(25), z12), z3);
  b = __dmul_rn(__dmul_rn(c.kr(25), z1), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(26), z12), z3);
  b = __dmul_rn(__dmul_rn(c.kr(26), z11), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d11 = __dadd_rn(d11, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(27), z3), z3);
  b = __dmul_rn(c.kr(27), z11);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(c.kf(28), z11);
  b = __dmul_rn(c.kr(28), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(29), z11), z3);
  b = __dmul_rn(__dmul_rn(c.kr(29), z1), z3);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(30), z11), z4);
  b = __dmul_rn(__dmul_rn(c.kr(30), z1), z4);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(31), z11), z3);
  b = __dmul_rn(__dmul_rn(c.kr(31), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(32), z11), z12);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(32), z1), z1), z3);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d11 = __dsub_rn(d11, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(33), z9), z11);
  b = __dmul_rn(__dmul_rn(c.kr(33), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(34), z9), z1);
  b = __dmul_rn(__dmul_rn(c.kr(34), z3), z11);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(35), z9), z1);
  b = __dmul_rn(__dmul_rn(c.kr(35), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(c.kf(36), z9);
  b = __dmul_rn(c.kr(36), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(37), z9), z2);
  b = __dmul_rn(__dmul_rn(c.kr(37), z3), z2);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(38), z9), z12);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(38), z1), z3), z3);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(39), z9), z12);
  b = __dmul_rn(__dmul_rn(c.kr(39), z1), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(40), z0), z11);
  b = __dmul_rn(__dmul_rn(c.kr(40), z4), z7);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(41), z4), z11);
  b = __dmul_rn(__dmul_rn(c.kr(41), z5), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(42), z4), z11);
  b = __dmul_rn(c.kr(42), z7);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(43), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(43), z6), z11);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(44), z5), z11);
  b = __dmul_rn(__dmul_rn(c.kr(44), z3), z7);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(45), z12), z4);
  b = __dmul_rn(__dmul_rn(c.kr(45), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(46), z12), z5);
  b = __dmul_rn(__dmul_rn(c.kr(46), z7), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(47), z12), z7);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(47), z5), z1), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(48), z4), z7);
  b = __dmul_rn(__dmul_rn(c.kr(48), z6), z9);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(49), z9), z0);
  b = __dmul_rn(__dmul_rn(c.kr(49), z5), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(50), z9), z6);
  b = __dmul_rn(__dmul_rn(c.kr(50), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(51), z3), z4);
  b = __dmul_rn(c.kr(51), z10);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d10 = __dadd_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(52), z10), z1);
  b = __dmul_rn(__dmul_rn(c.kr(52), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(53), z10), z2);
  b = __dmul_rn(__dmul_rn(c.kr(53), z5), z2);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(54), z10), z6);
  b = __dmul_rn(__dmul_rn(c.kr(54), z5), z6);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(55), z10), z0);
  b = __dmul_rn(__dmul_rn(c.kr(55), z5), z0);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(56), z10), z5);
  b = __dmul_rn(__dmul_rn(c.kr(56), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(57), z10), z4);
  b = __dmul_rn(__dmul_rn(c.kr(57), z5), z4);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(58), z10), z3);
  b = __dmul_rn(__dmul_rn(c.kr(58), z5), z3);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(59), z10), z0);
  b = __dmul_rn(__dmul_rn(c.kr(59), z6), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(60), z10), z1);
  b = __dmul_rn(__dmul_rn(c.kr(60), z12), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d10 = __dsub_rn(d10, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(61), z10), z1);
  b = __dmul_rn(__dmul_rn(c.kr(61), z7), z3);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d7 = __dadd_rn(d7, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(62), z10), z6);
  b = __dmul_rn(__dmul_rn(c.kr(62), z8), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(63), z4), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(63), z0), z1);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(64), z4), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(64), z5), z5);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(65), z4), z1), z3);
  b = __dmul_rn(__dmul_rn(c.kr(65), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(66), z4), z1), z5);
  b = __dmul_rn(__dmul_rn(c.kr(66), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  c.zd(0) = d0;
  c.zd(1) = d1;
  c.zd(2) = d2;
  c.zd(3) = d3;
  c.zd(4) = d4;
  c.zd(5) = d5;
  c.zd(6) = d6;
  c.zd(7) = d7;
  c.zd(8) = d8;
  c.zd(9) = d9;
  c.zd(10) = d10;
  c.zd(11) = d11;
  c.zd(12) = d12;
}

constexpr int kFullN = 13, kFullR = 71;
constexpr int kFullLeft[71][3] = {
    {4, 4, -1},
    {4, 4, 0},
    {4, 4, 2},
    {4, 4, 4},
    {3, 3, -1},
    {3, 4, -1},
    {6, -1, -1},
    {6, 6, -1},
    {4, 1, -1},
    {8, -1, -1},
    {3, 0, -1},
    {4, 1, -1},
    {0, 5, -1},
    {5, 5, -1},
    {7, 3, -1},
    {4, 7, -1},
    {6, 3, -1},
    {0, 1, -1},
    {7, 5, -1},
    {7, 5, -1},
    {7, 7, -1},
    {7, 7, -1},
    {8, 4, -1},
    {8, 4, -1},
    {8, 3, -1},
    {8, 5, -1},
    {8, 5, -1},
    {1, 3, -1},
    {1, 3, -1},
    {12, 3, -1},
    {12, 3, -1},
    {3, 3, -1},
    {11, -1, -1},
    {11, 3, -1},
    {11, 4, -1},
    {11, 3, -1},
    {11, 12, -1},
    {9, 11, -1},
    {9, 1, -1},
    {9, 1, -1},
    {9, -1, -1},
    {9, 2, -1},
    {9, 12, -1},
    {9, 12, -1},
    {0, 11, -1},
    {4, 11, -1},
    {4, 11, -1},
    {7, 5, -1},
    {5, 11, -1},
    {12, 4, -1},
    {12, 5, -1},
    {12, 7, -1},
    {4, 7, -1},
    {9, 0, -1},
    {9, 6, -1},
    {3, 4, -1},
    {10, 1, -1},
    {10, 2, -1},
    {10, 6, -1},
    {10, 0, -1},
    {10, 5, -1},
    {10, 4, -1},
    {10, 3, -1},
    {10, 0, -1},
    {10, 1, -1},
    {10, 1, -1},
    {10, 6, -1},
    {4, 1, 4},
    {4, 1, 4},
    {4, 1, 3},
    {4, 1, 5},
};
constexpr int kFullRight[71][3] = {
    {0, -1, -1},
    {0, 0, -1},
    {0, 2, -1},
    {0, 4, -1},
    {1, -1, -1},
    {5, -1, -1},
    {4, 5, -1},
    {4, 5, 6},
    {7, -1, -1},
    {5, 5, -1},
    {5, 4, -1},
    {5, 3, -1},
    {6, 4, -1},
    {6, 3, -1},
    {5, 1, -1},
    {5, 5, -1},
    {4, 7, -1},
    {4, 7, -1},
    {6, 1, -1},
    {6, 1, -1},
    {8, 1, -1},
    {8, 1, -1},
    {7, 0, -1},
    {6, 5, -1},
    {7, 5, -1},
    {7, 6, -1},
    {7, 6, -1},
    {12, -1, -1},
    {12, -1, -1},
    {1, 1, -1},
    {11, 1, -1},
    {11, -1, -1},
    {1, -1, -1},
    {1, 3, -1},
    {1, 4, -1},
    {3, 1, -1},
    {1, 1, 3},
    {3, 1, -1},
    {3, 11, -1},
    {3, 1, -1},
    {3, -1, -1},
    {3, 2, -1},
    {1, 3, 3},
    {1, 1, -1},
    {4, 7, -1},
    {5, 3, -1},
    {7, -1, -1},
    {6, 11, -1},
    {3, 7, -1},
    {5, 1, -1},
    {7, 1, -1},
    {5, 1, 1},
    {6, 9, -1},
    {5, 4, -1},
    {5, 5, -1},
    {10, -1, -1},
    {5, 1, -1},
    {5, 2, -1},
    {5, 6, -1},
    {5, 0, -1},
    {5, 5, -1},
    {5, 4, -1},
    {5, 3, -1},
    {6, 4, -1},
    {12, 4, -1},
    {7, 3, -1},
    {8, 4, -1},
    {0, 1, -1},
    {5, 5, -1},
    {5, 1, -1},
    {6, 1, -1},
};
constexpr int kFullNupd[71] = {3, 5, 5, 5, 3, 3, 3, 5, 3, 3, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 3, 3, 4, 4, 3, 2, 4, 4, 4, 5, 4, 4, 4, 2, 4, 5, 4, 4, 4, 3, 4, 4, 4, 4, 5, 4, 4, 4, 3, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 5, 5, 5, 5};
constexpr int kFullUpdK[71][6] = {
    {0, 4, 4, 0, 0, 0},
    {0, 0, 0, 4, 4, 0},
    {0, 2, 2, 4, 4, 0},
    {0, 4, 4, 4, 4, 0},
    {1, 3, 3, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {4, 5, 6, 0, 0, 0},
    {4, 5, 6, 6, 6, 0},
    {1, 4, 7, 0, 0, 0},
    {5, 5, 8, 0, 0, 0},
    {0, 3, 4, 5, 0, 0},
    {1, 3, 4, 5, 0, 0},
    {0, 4, 5, 6, 0, 0},
    {3, 5, 5, 6, 0, 0},
    {1, 3, 5, 7, 0, 0},
    {4, 5, 5, 7, 0, 0},
    {3, 4, 6, 7, 0, 0},
    {0, 1, 4, 7, 0, 0},
    {1, 5, 6, 7, 0, 0},
    {1, 5, 6, 7, 0, 0},
    {1, 7, 7, 8, 0, 0},
    {1, 7, 7, 8, 0, 0},
    {0, 4, 7, 8, 0, 0},
    {4, 5, 6, 8, 0, 0},
    {3, 5, 7, 8, 0, 0},
    {5, 6, 7, 8, 0, 0},
    {5, 6, 7, 8, 0, 0},
    {1, 3, 12, 0, 0, 0},
    {1, 3, 12, 0, 0, 0},
    {1, 1, 3, 12, 0, 0},
    {1, 3, 11, 12, 0, 0},
    {3, 3, 11, 0, 0, 0},
    {1, 11, 0, 0, 0, 0},
    {1, 3, 3, 11, 0, 0},
    {1, 4, 4, 11, 0, 0},
    {1, 3, 3, 11, 0, 0},
    {1, 1, 3, 11, 12, 0},
    {1, 3, 9, 11, 0, 0},
    {1, 3, 9, 11, 0, 0},
    {1, 1, 3, 9, 0, 0},
    {3, 9, 0, 0, 0, 0},
    {2, 2, 3, 9, 0, 0},
    {1, 3, 3, 9, 12, 0},
    {1, 1, 9, 12, 0, 0},
    {0, 4, 7, 11, 0, 0},
    {3, 4, 5, 11, 0, 0},
    {4, 7, 11, 0, 0, 0},
    {5, 6, 7, 11, 0, 0},
    {3, 5, 7, 11, 0, 0},
    {1, 4, 5, 12, 0, 0},
    {1, 5, 7, 12, 0, 0},
    {1, 1, 5, 7, 12, 0},
    {4, 6, 7, 9, 0, 0},
    {0, 4, 5, 9, 0, 0},
    {5, 5, 6, 9, 0, 0},
    {3, 4, 10, 0, 0, 0},
    {1, 1, 5, 10, 0, 0},
    {2, 2, 5, 10, 0, 0},
    {5, 6, 6, 10, 0, 0},
    {0, 0, 5, 10, 0, 0},
    {5, 5, 5, 10, 0, 0},
    {4, 4, 5, 10, 0, 0},
    {3, 3, 5, 10, 0, 0},
    {0, 4, 6, 10, 0, 0},
    {1, 4, 10, 12, 0, 0},
    {1, 3, 7, 10, 0, 0},
    {4, 6, 8, 10, 0, 0},
    {0, 1, 1, 4, 4, 0},
    {1, 4, 4, 5, 5, 0},
    {1, 1, 3, 4, 5, 0},
    {1, 1, 4, 5, 6, 0},
};
constexpr int kFullUpdProd[71][6] = {
    {1, 0, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 0, 0, 1, 0},
    {1, 0, 0, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 1, 0, 0, 1, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 0, 0, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 1, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 1, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 0, 1, 1, 0},
    {0, 1, 0, 0, 1, 0},
    {0, 1, 0, 0, 1, 0},
};

// zd = dC/dt at z (shared scratch in, shared scratch out)
template <class S>
__device__ __forceinline__ void full_rhs(S& c) {
  const double z0 = c.z(0);
  const double z1 = c.z(1);
  const double z2 = c.z(2);
  const double z3 = c.z(3);
  const double z4 = c.z(4);
  const double z5 = c.z(5);
  const double z6 = c.z(6);
  const double z7 = c.z(7);
  const double z8 = c.z(8);
  const double z9 = c.z(9);
  const double z10 = c.z(10);
  const double z11 = c.z(11);
  const double z12 = c.z(12);
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0, d9 = 0.0, d10 = 0.0, d11 = 0.0, d12 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z4), z4);
  b = __dmul_rn(c.kr(0), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(1), z4), z4), z0);
  b = __dmul_rn(__dmul_rn(c.kr(1), z0), z0);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(2), z4), z4), z2);
  b = __dmul_rn(__dmul_rn(c.kr(2), z0), z2);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(3), z4), z4), z4);
  b = __dmul_rn(__dmul_rn(c.kr(3), z0), z4);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(4), z3), z3);
  b = __dmul_rn(c.kr(4), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z3), z4);
  b = __dmul_rn(c.kr(5), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(c.kf(6), z6);
  b = __dmul_rn(__dmul_rn(c.kr(6), z4), z5);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(7), z6), z6);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(7), z4), z5), z6);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z4), z1);
  b = __dmul_rn(c.kr(8), z7);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(c.kf(9), z8);
  b = __dmul_rn(__dmul_rn(c.kr(9), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(10), z3), z0);
  b = __dmul_rn(__dmul_rn(c.kr(10), z5), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z4), z1);
  b = __dmul_rn(__dmul_rn(c.kr(11), z5), z3);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(12), z0), z5);
  b = __dmul_rn(__dmul_rn(c.kr(12), z6), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(13), z5), z5);
  b = __dmul_rn(__dmul_rn(c.kr(13), z6), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(14), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(14), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z4), z7);
  b = __dmul_rn(__dmul_rn(c.kr(15), z5), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z6), z3);
  b = __dmul_rn(__dmul_rn(c.kr(16), z4), z7);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z0), z1);
  b = __dmul_rn(__dmul_rn(c.kr(17), z4), z7);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(18), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(19), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(19), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z7), z7);
  b = __dmul_rn(__dmul_rn(c.kr(20), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z7), z7);
  b = __dmul_rn(__dmul_rn(c.kr(21), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(22), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(22), z7), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(23), z6), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(24), z8), z3);
  b = __dmul_rn(__dmul_rn(c.kr(24), z7), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(25), z8), z5);
  b = __dmul_rn(__dmul_rn(c.kr(25), z7), z6);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(26), z8), z5);
  b = __dmul_rn(__dmul_rn(c.kr(26), z7), z6);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(27), z1), z3);
  b = __dmul_rn(c.kr(27), z12);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(28), z1), z3);
  b = __dmul_rn(c.kr(28), z12);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(29), z12), z3);
  b = __dmul_rn(__dmul_rn(c.kr(29), z1), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(30), z12), z3);
  b = __dmul_rn(__dmul_rn(c.kr(30), z11), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d11 = __dadd_rn(d11, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(31), z3), z3);
  b = __dmul_rn(c.kr(31), z11);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(c.kf(32), z11);
  b = __dmul_rn(c.kr(32), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(33), z11), z3);
  b = __dmul_rn(__dmul_rn(c.kr(33), z1), z3);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(34), z11), z4);
  b = __dmul_rn(__dmul_rn(c.kr(34), z1), z4);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(35), z11), z3);
  b = __dmul_rn(__dmul_rn(c.kr(35), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(36), z11), z12);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(36), z1), z1), z3);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d11 = __dsub_rn(d11, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(37), z9), z11);
  b = __dmul_rn(__dmul_rn(c.kr(37), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(38), z9), z1);
  b = __dmul_rn(__dmul_rn(c.kr(38), z3), z11);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(39), z9), z1);
  b = __dmul_rn(__dmul_rn(c.kr(39), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(c.kf(40), z9);
  b = __dmul_rn(c.kr(40), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(41), z9), z2);
  b = __dmul_rn(__dmul_rn(c.kr(41), z3), z2);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(42), z9), z12);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(42), z1), z3), z3);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(43), z9), z12);
  b = __dmul_rn(__dmul_rn(c.kr(43), z1), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(44), z0), z11);
  b = __dmul_rn(__dmul_rn(c.kr(44), z4), z7);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(45), z4), z11);
  b = __dmul_rn(__dmul_rn(c.kr(45), z5), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(46), z4), z11);
  b = __dmul_rn(c.kr(46), z7);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(47), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(47), z6), z11);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(48), z5), z11);
  b = __dmul_rn(__dmul_rn(c.kr(48), z3), z7);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(49), z12), z4);
  b = __dmul_rn(__dmul_rn(c.kr(49), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(50), z12), z5);
  b = __dmul_rn(__dmul_rn(c.kr(50), z7), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(51), z12), z7);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(51), z5), z1), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(52), z4), z7);
  b = __dmul_rn(__dmul_rn(c.kr(52), z6), z9);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(53), z9), z0);
  b = __dmul_rn(__dmul_rn(c.kr(53), z5), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(54), z9), z6);
  b = __dmul_rn(__dmul_rn(c.kr(54), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(55), z3), z4);
  b = __dmul_rn(c.kr(55), z10);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d10 = __dadd_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(56), z10), z1);
  b = __dmul_rn(__dmul_rn(c.kr(56), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(57), z10), z2);
  b = __dmul_rn(__dmul_rn(c.kr(57), z5), z2);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(58), z10), z6);
  b = __dmul_rn(__dmul_rn(c.kr(58), z5), z6);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(59), z10), z0);
  b = __dmul_rn(__dmul_rn(c.kr(59), z5), z0);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(60), z10), z5);
  b = __dmul_rn(__dmul_rn(c.kr(60), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(61), z10), z4);
  b = __dmul_rn(__dmul_rn(c.kr(61), z5), z4);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(62), z10), z3);
  b = __dmul_rn(__dmul_rn(c.kr(62), z5), z3);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(63), z10), z0);
  b = __dmul_rn(__dmul_rn(c.kr(63), z6), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(64), z10), z1);
  b = __dmul_rn(__dmul_rn(c.kr(64), z12), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d10 = __dsub_rn(d10, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(65), z10), z1);
  b = __dmul_rn(__dmul_rn(c.kr(65), z7), z3);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d7 = __dadd_rn(d7, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(66), z10), z6);
  b = __dmul_rn(__dmul_rn(c.kr(66), z8), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(67), z4), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(67), z0), z1);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(68), z4), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(68), z5), z5);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(69), z4), z1), z3);
  b = __dmul_rn(__dmul_rn(c.kr(69), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(70), z4), z1), z5);
  b = __dmul_rn(__dmul_rn(c.kr(70), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  c.zd(0) = d0;
  c.zd(1) = d1;
  c.zd(2) = d2;
  c.zd(3) = d3;
  c.zd(4) = d4;
  c.zd(5) = d5;
  c.zd(6) = d6;
  c.zd(7) = d7;
  c.zd(8) = d8;
  c.zd(9) = d9;
  c.zd(10) = d10;
  c.zd(11) = d11;
  c.zd(12) = d12;
}

// Column J of I + factor * J: v[i] = A(i+1, J+1), each element's terms in
// reaction order.
template <int J, class S, typename LUT>
__device__ __forceinline__ void spec_column(const S& c, double factor, LUT (&v)[13]) {
  const double msf = -factor;
  double d;
  if constexpr (J == 0) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z7 = c.z(7), z9 = c.z(9), z10 = c.z(10), z11 = c.z(11);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kr(0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(1), z4), z4), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z0), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z0), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(2), z2), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z4), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(10), z3), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(12), z5), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z1), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z7), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(40), z11), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(49), z9), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(55), z10), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(55), z5), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(59), z10), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(63), z1), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a0 = a0 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 1) {
    const double z0 = c.z(0), z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z9 = c.z(9), z10 = c.z(10), z11 = c.z(11);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kr(4), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z4), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z4), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z5), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(18), z6), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z8), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(24), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(25), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(25), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(26), z11), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(c.kr(28), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(29), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(30), z4), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(31), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(32), z1), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(32), z1), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(33), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(34), z9), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(35), z9), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(35), z3), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(38), z3), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(39), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(39), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(45), z5), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(46), z7), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(47), z5), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(47), z5), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(52), z10), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(52), z5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(60), z10), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(61), z10), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(63), z4), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(63), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(64), z4), z4), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(65), z4), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(65), z5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(66), z4), z5), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(66), z6), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a1 = a1 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 2) {
    const double z0 = c.z(0), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z9 = c.z(9), z10 = c.z(10);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(2), z4), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(2), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(37), z9), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(37), z3), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(53), z10), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(53), z5), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a2 = a2 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 3) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z10 = c.z(10), z11 = c.z(11), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(4), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kf(4), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z4), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(10), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z6), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(14), z7), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(16), z6), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(22), z8), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(24), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(25), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(26), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(27), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(27), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(29), z11), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(29), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(31), z11), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(31), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(32), z1), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(33), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(34), z11), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(35), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(c.kr(36), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(37), z2), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(38), z1), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(38), z1), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(41), z5), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(44), z7), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(51), z4), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(58), z10), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(58), z5), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(61), z7), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(65), z4), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a3 = a3 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 4) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z10 = c.z(10), z11 = c.z(11), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(0), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(1), z4), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(1), z4), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(2), z4), z2), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(2), z4), z2), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(3), z4), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(3), z4), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(3), z4), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(6), z5), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(7), z5), z6), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z5), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z6), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z7), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(16), z7), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z7), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z8), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(21), z8), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(30), z11), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(30), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(40), z7), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(41), z11), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(42), z11), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(45), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(48), z7), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(49), z5), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(51), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(57), z10), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(57), z5), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(59), z6), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(60), z12), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(62), z8), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(63), z1), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(63), z4), z1), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(64), z1), z4), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(64), z4), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(65), z1), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(66), z1), z5), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a4 = a4 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 5) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z10 = c.z(10), z11 = c.z(11), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kr(5), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(6), z4), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(7), z4), z6), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(9), z5), msf);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(9), z5), msf);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z3), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(12), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(13), z5), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(13), z5), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(15), z5), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(15), z5), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z7), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z6), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(22), z7), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(23), z8), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(41), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(43), z7), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(44), z11), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(45), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(46), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(47), z1), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(49), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(50), z5), msf);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(50), z5), msf);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(52), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(53), z2), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(54), z6), msf);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(55), z0), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(56), z10), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(56), z5), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(56), z5), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(57), z4), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(58), z3), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(64), z5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(64), z5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(65), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(66), z4), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a5 = a5 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 6) {
    const double z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z9 = c.z(9), z10 = c.z(10), z11 = c.z(11);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kf(6), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(7), z6), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(7), z6), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(7), z4), z5), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(16), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(18), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z5), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z7), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(43), z11), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(48), z9), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(50), z9), factor);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(54), z10), factor);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(54), z5), msf);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(59), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(62), z10), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(66), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a6 = a6 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 7) {
    const double z0 = c.z(0), z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kr(8), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(14), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(16), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z5), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(19), z7), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(19), z7), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(22), z5), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z6), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(40), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(c.kr(42), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(43), z5), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(44), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(46), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(47), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(48), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(61), z3), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a7 = a7 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 8) {
    const double z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kf(9), factor);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z4), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(21), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(22), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(23), z5), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(62), z4), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a8 = a8 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 9) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z6 = c.z(6), z11 = c.z(11), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(33), z11), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(34), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(35), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(c.kf(36), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(37), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(38), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(39), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(48), z6), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(49), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(50), z6), factor);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a9 = a9 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 10) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kr(51), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(52), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(53), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(54), z6), factor);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(55), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(56), z5), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(57), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(58), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(59), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(60), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(61), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(62), z6), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a10 = a10 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 11) {
    const double z0 = c.z(0), z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z9 = c.z(9), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(26), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(c.kr(27), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(c.kf(28), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(29), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(30), z4), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(31), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(32), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(33), z9), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(34), z3), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(40), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(41), z4), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(42), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(43), z6), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(44), z5), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a11 = a11 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
  if constexpr (J == 12) {
    const double z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z7 = c.z(7), z9 = c.z(9), z11 = c.z(11);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0;
    d = __dmul_rn(c.kr(24), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(25), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(26), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(32), z11), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(38), z9), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(39), z9), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(45), z4), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(46), z5), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(47), z7), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(60), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    a12 = a12 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12;
  }
}

}  // namespace gen_konnov
}  // namespace nrg
