// Generated by nrg_b200/gen_mech.py from ZHANG.txt: do not edit.
// Straight-line right-hand side and analytic iteration matrix over the
// 8 reacting species and 25 distinct reactions, and the right-hand side
// over all 9 species and 28 reactions; same operation order as the
// table-driven loops in chem_bdf.cuh, with the same explicitly rounded
// (never fused) operations.
#pragma once

namespace nrg {
namespace gen_zhang {

constexpr int kSpecN = 8, kSpecR = 25;
constexpr int kSpecLeft[25][3] = {
    {3, 1, -1},
    {2, 0, -1},
    {4, 0, -1},
    {4, 4, -1},
    {0, -1, -1},
    {2, 2, -1},
    {2, 3, -1},
    {5, -1, -1},
    {5, 5, -1},
    {3, 1, -1},
    {6, 3, -1},
    {6, 3, -1},
    {5, 2, -1},
    {6, 2, -1},
    {6, 4, -1},
    {6, 6, -1},
    {7, -1, -1},
    {7, 3, -1},
    {7, 3, -1},
    {7, 2, -1},
    {7, 4, -1},
    {3, 1, 3},
    {3, 1, 3},
    {3, 1, 2},
    {3, 1, 4},
};
constexpr int kSpecRight[25][3] = {
    {2, 4, -1},
    {4, 3, -1},
    {3, 5, -1},
    {5, 2, -1},
    {3, 3, -1},
    {1, -1, -1},
    {4, -1, -1},
    {3, 4, -1},
    {3, 4, 5},
    {6, -1, -1},
    {0, 1, -1},
    {4, 4, -1},
    {3, 6, -1},
    {4, 1, -1},
    {5, 1, -1},
    {7, 1, -1},
    {4, 4, -1},
    {5, 4, -1},
    {6, 0, -1},
    {4, 6, -1},
    {5, 6, -1},
    {0, 1, -1},
    {4, 4, -1},
    {4, 1, -1},
    {5, 1, -1},
};
constexpr int kSpecNupd[25] = {4, 4, 4, 4, 3, 3, 3, 3, 5, 3, 4, 4, 4, 4, 4, 4, 3, 4, 4, 4, 4, 5, 5, 5, 5};
constexpr int kSpecUpdK[25][6] = {
    {1, 2, 3, 4, 0, 0},
    {0, 2, 3, 4, 0, 0},
    {0, 3, 4, 5, 0, 0},
    {2, 4, 4, 5, 0, 0},
    {0, 3, 3, 0, 0, 0},
    {1, 2, 2, 0, 0, 0},
    {2, 3, 4, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {3, 4, 5, 5, 5, 0},
    {1, 3, 6, 0, 0, 0},
    {0, 1, 3, 6, 0, 0},
    {3, 4, 4, 6, 0, 0},
    {2, 3, 5, 6, 0, 0},
    {1, 2, 4, 6, 0, 0},
    {1, 4, 5, 6, 0, 0},
    {1, 6, 6, 7, 0, 0},
    {4, 4, 7, 0, 0, 0},
    {3, 4, 5, 7, 0, 0},
    {0, 3, 6, 7, 0, 0},
    {2, 4, 6, 7, 0, 0},
    {4, 5, 6, 7, 0, 0},
    {0, 1, 1, 3, 3, 0},
    {1, 3, 3, 4, 4, 0},
    {1, 1, 2, 3, 4, 0},
    {1, 1, 3, 4, 5, 0},
};
constexpr int kSpecUpdProd[25][6] = {
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 1, 0, 0, 1, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
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
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z3), z1);
  b = __dmul_rn(__dmul_rn(c.kr(0), z2), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d2 = __dadd_rn(d2, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(1), z2), z0);
  b = __dmul_rn(__dmul_rn(c.kr(1), z4), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d2 = __dsub_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(2), z4), z0);
  b = __dmul_rn(__dmul_rn(c.kr(2), z3), z5);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(3), z4), z4);
  b = __dmul_rn(__dmul_rn(c.kr(3), z5), z2);
  q = __dsub_rn(f, b);
  d2 = __dadd_rn(d2, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(c.kf(4), z0);
  b = __dmul_rn(__dmul_rn(c.kr(4), z3), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z2), z2);
  b = __dmul_rn(c.kr(5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d2 = __dsub_rn(d2, q);
  d2 = __dsub_rn(d2, q);
  f = __dmul_rn(__dmul_rn(c.kf(6), z2), z3);
  b = __dmul_rn(c.kr(6), z4);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(c.kf(7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(7), z3), z4);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z5), z5);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(8), z3), z4), z5);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d5 = __dsub_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(9), z3), z1);
  b = __dmul_rn(c.kr(9), z6);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(10), z6), z3);
  b = __dmul_rn(__dmul_rn(c.kr(10), z0), z1);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z6), z3);
  b = __dmul_rn(__dmul_rn(c.kr(11), z4), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(12), z5), z2);
  b = __dmul_rn(__dmul_rn(c.kr(12), z3), z6);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(13), z6), z2);
  b = __dmul_rn(__dmul_rn(c.kr(13), z4), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d2 = __dsub_rn(d2, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(14), z6), z4);
  b = __dmul_rn(__dmul_rn(c.kr(14), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z6), z6);
  b = __dmul_rn(__dmul_rn(c.kr(15), z7), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dsub_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(c.kf(16), z7);
  b = __dmul_rn(__dmul_rn(c.kr(16), z4), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(17), z5), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(18), z6), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(19), z7), z2);
  b = __dmul_rn(__dmul_rn(c.kr(19), z4), z6);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z7), z4);
  b = __dmul_rn(__dmul_rn(c.kr(20), z5), z6);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(21), z3), z1), z3);
  b = __dmul_rn(__dmul_rn(c.kr(21), z0), z1);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(22), z3), z1), z3);
  b = __dmul_rn(__dmul_rn(c.kr(22), z4), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(23), z3), z1), z2);
  b = __dmul_rn(__dmul_rn(c.kr(23), z4), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d2 = __dsub_rn(d2, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(24), z3), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(24), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  c.zd(0) = d0;
  c.zd(1) = d1;
  c.zd(2) = d2;
  c.zd(3) = d3;
  c.zd(4) = d4;
  c.zd(5) = d5;
  c.zd(6) = d6;
  c.zd(7) = d7;
}

constexpr int kFullN = 9, kFullR = 28;
constexpr int kFullLeft[28][3] = {
    {4, 1, -1},
    {3, 0, -1},
    {5, 0, -1},
    {5, 5, -1},
    {0, -1, -1},
    {3, 3, -1},
    {3, 4, -1},
    {6, -1, -1},
    {6, 6, -1},
    {4, 1, -1},
    {7, 4, -1},
    {7, 4, -1},
    {6, 3, -1},
    {7, 3, -1},
    {7, 5, -1},
    {7, 5, -1},
    {7, 7, -1},
    {7, 7, -1},
    {8, -1, -1},
    {8, 4, -1},
    {8, 4, -1},
    {8, 3, -1},
    {8, 5, -1},
    {8, 5, -1},
    {4, 1, 4},
    {4, 1, 4},
    {4, 1, 3},
    {4, 1, 5},
};
constexpr int kFullRight[28][3] = {
    {3, 5, -1},
    {5, 4, -1},
    {4, 6, -1},
    {6, 3, -1},
    {4, 4, -1},
    {1, -1, -1},
    {5, -1, -1},
    {4, 5, -1},
    {4, 5, 6},
    {7, -1, -1},
    {0, 1, -1},
    {5, 5, -1},
    {4, 7, -1},
    {5, 1, -1},
    {6, 1, -1},
    {6, 1, -1},
    {8, 1, -1},
    {8, 1, -1},
    {5, 5, -1},
    {6, 5, -1},
    {7, 0, -1},
    {5, 7, -1},
    {6, 7, -1},
    {6, 7, -1},
    {0, 1, -1},
    {5, 5, -1},
    {5, 1, -1},
    {6, 1, -1},
};
constexpr int kFullNupd[28] = {4, 4, 4, 4, 3, 3, 3, 3, 5, 3, 4, 4, 4, 4, 4, 4, 4, 4, 3, 4, 4, 4, 4, 4, 5, 5, 5, 5};
constexpr int kFullUpdK[28][6] = {
    {1, 3, 4, 5, 0, 0},
    {0, 3, 4, 5, 0, 0},
    {0, 4, 5, 6, 0, 0},
    {3, 5, 5, 6, 0, 0},
    {0, 4, 4, 0, 0, 0},
    {1, 3, 3, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {4, 5, 6, 0, 0, 0},
    {4, 5, 6, 6, 6, 0},
    {1, 4, 7, 0, 0, 0},
    {0, 1, 4, 7, 0, 0},
    {4, 5, 5, 7, 0, 0},
    {3, 4, 6, 7, 0, 0},
    {1, 3, 5, 7, 0, 0},
    {1, 5, 6, 7, 0, 0},
    {1, 5, 6, 7, 0, 0},
    {1, 7, 7, 8, 0, 0},
    {1, 7, 7, 8, 0, 0},
    {5, 5, 8, 0, 0, 0},
    {4, 5, 6, 8, 0, 0},
    {0, 4, 7, 8, 0, 0},
    {3, 5, 7, 8, 0, 0},
    {5, 6, 7, 8, 0, 0},
    {5, 6, 7, 8, 0, 0},
    {0, 1, 1, 4, 4, 0},
    {1, 4, 4, 5, 5, 0},
    {1, 1, 3, 4, 5, 0},
    {1, 1, 4, 5, 6, 0},
};
constexpr int kFullUpdProd[28][6] = {
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 1, 0, 0, 1, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
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
  const double z3 = c.z(3);
  const double z4 = c.z(4);
  const double z5 = c.z(5);
  const double z6 = c.z(6);
  const double z7 = c.z(7);
  const double z8 = c.z(8);
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z4), z1);
  b = __dmul_rn(__dmul_rn(c.kr(0), z3), z5);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(1), z3), z0);
  b = __dmul_rn(__dmul_rn(c.kr(1), z5), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(2), z5), z0);
  b = __dmul_rn(__dmul_rn(c.kr(2), z4), z6);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(3), z5), z5);
  b = __dmul_rn(__dmul_rn(c.kr(3), z6), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(c.kf(4), z0);
  b = __dmul_rn(__dmul_rn(c.kr(4), z4), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z3), z3);
  b = __dmul_rn(c.kr(5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d3 = __dsub_rn(d3, q);
  f = __dmul_rn(__dmul_rn(c.kf(6), z3), z4);
  b = __dmul_rn(c.kr(6), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(c.kf(7), z6);
  b = __dmul_rn(__dmul_rn(c.kr(7), z4), z5);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z6), z6);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(8), z4), z5), z6);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(9), z4), z1);
  b = __dmul_rn(c.kr(9), z7);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(10), z7), z4);
  b = __dmul_rn(__dmul_rn(c.kr(10), z0), z1);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z7), z4);
  b = __dmul_rn(__dmul_rn(c.kr(11), z5), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(12), z6), z3);
  b = __dmul_rn(__dmul_rn(c.kr(12), z4), z7);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(13), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(13), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(14), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(14), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(15), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z7), z7);
  b = __dmul_rn(__dmul_rn(c.kr(16), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z7), z7);
  b = __dmul_rn(__dmul_rn(c.kr(17), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(c.kf(18), z8);
  b = __dmul_rn(__dmul_rn(c.kr(18), z5), z5);
  q = __dsub_rn(f, b);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(19), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(19), z6), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(20), z7), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z8), z3);
  b = __dmul_rn(__dmul_rn(c.kr(21), z5), z7);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(22), z8), z5);
  b = __dmul_rn(__dmul_rn(c.kr(22), z6), z7);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z8), z5);
  b = __dmul_rn(__dmul_rn(c.kr(23), z6), z7);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(24), z4), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(24), z0), z1);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(25), z4), z1), z4);
  b = __dmul_rn(__dmul_rn(c.kr(25), z5), z5);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(26), z4), z1), z3);
  b = __dmul_rn(__dmul_rn(c.kr(26), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(27), z4), z1), z5);
  b = __dmul_rn(__dmul_rn(c.kr(27), z6), z1);
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
}

// Column J of I + factor * J: v[i] = A(i+1, J+1), each element's terms in
// reaction order.
template <int J, class S, typename LUT>
__device__ __forceinline__ void spec_column(const S& c, double factor, LUT (&v)[8]) {
  const double msf = -factor;
  double d;
  if constexpr (J == 0) {
    const double z1 = c.z(1), z2 = c.z(2), z4 = c.z(4), z6 = c.z(6);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(1), z2), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(2), z4), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(c.kf(4), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z1), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(18), z6), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z1), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a0 = a0 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 1) {
    const double z0 = c.z(0), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z7 = c.z(7);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(c.kr(5), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    d = __dmul_rn(__dmul_rn(c.kf(9), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z4), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z5), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(15), z7), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(21), z3), z3), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(22), z3), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(23), z3), z2), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(24), z3), z4), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(24), z5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a1 = a1 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 2) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(0), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(1), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z5), msf);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z2), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z2), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    d = __dmul_rn(__dmul_rn(c.kf(6), z3), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(12), z5), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(13), z6), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(19), z7), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(23), z3), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a2 = a2 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 3) {
    const double z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z4), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(2), z5), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(4), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kr(4), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kf(6), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(7), z4), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(8), z4), z5), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(9), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(10), z6), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z6), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z6), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z7), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z7), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(21), z1), z3), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(21), z3), z1), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(22), z1), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(22), z3), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(23), z1), z2), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(24), z1), z4), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a3 = a3 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 4) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(0), z2), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(2), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(3), z4), factor);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(3), z4), factor);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(c.kr(6), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(7), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(8), z3), z5), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(14), z6), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(16), z4), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(16), z4), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z5), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z6), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z7), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(22), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(22), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kf(24), z3), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a4 = a4 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 5) {
    const double z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(2), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z2), msf);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(c.kf(7), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z5), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z5), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(8), z3), z4), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(12), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z6), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(24), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a5 = a5 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 6) {
    const double z0 = c.z(0), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(c.kr(9), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(10), z3), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z3), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(13), z2), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(14), z4), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z6), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z6), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(18), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z4), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z5), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a6 = a6 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
  if constexpr (J == 7) {
    const double z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(15), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(c.kf(16), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z3), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(19), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a7 = a7 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7;
  }
}

}  // namespace gen_zhang
}  // namespace nrg
