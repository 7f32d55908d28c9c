// Generated by nrg_b200/gen_mech.py from TEREZA.txt: do not edit.
// Straight-line right-hand side and analytic iteration matrix over the
// 10 reacting species and 24 distinct reactions, and the right-hand side
// over all 10 species and 24 reactions; same operation order as the
// table-driven loops in chem_bdf.cuh, with the same explicitly rounded
// (never fused) operations.
#pragma once

namespace nrg {
namespace gen_tereza {

constexpr int kSpecN = 10, kSpecR = 24;
constexpr int kSpecLeft[24][3] = {
    {3, 1, -1},
    {9, 4, -1},
    {9, 3, -1},
    {9, 3, -1},
    {0, 4, -1},
    {8, 8, -1},
    {0, 8, -1},
    {7, 1, -1},
    {7, 8, -1},
    {7, 3, -1},
    {7, 3, -1},
    {7, 4, -1},
    {6, -1, -1},
    {1, -1, -1},
    {0, -1, -1},
    {4, 3, -1},
    {3, 4, -1},
    {5, 6, -1},
    {5, 0, -1},
    {5, 2, -1},
    {5, 8, -1},
    {5, 3, -1},
    {5, -1, -1},
    {5, 1, -1},
};
constexpr int kSpecRight[24][3] = {
    {4, 8, -1},
    {8, 1, -1},
    {8, 8, -1},
    {6, 4, -1},
    {3, 8, -1},
    {6, 4, -1},
    {6, 3, -1},
    {9, 9, -1},
    {6, 9, -1},
    {9, 0, -1},
    {6, 8, -1},
    {9, 8, -1},
    {3, 8, -1},
    {4, 4, -1},
    {3, 3, -1},
    {8, -1, -1},
    {-1, 5, -1},
    {8, 6, -1},
    {8, 0, -1},
    {8, 2, -1},
    {8, 8, -1},
    {8, 3, -1},
    {8, -1, -1},
    {8, 1, -1},
};
constexpr int kSpecNupd[24] = {4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 2, 4};
constexpr int kSpecUpdK[24][6] = {
    {1, 3, 4, 8, 0, 0},
    {1, 4, 8, 9, 0, 0},
    {3, 8, 8, 9, 0, 0},
    {3, 4, 6, 9, 0, 0},
    {0, 3, 4, 8, 0, 0},
    {4, 6, 8, 8, 0, 0},
    {0, 3, 6, 8, 0, 0},
    {1, 7, 9, 9, 0, 0},
    {6, 7, 8, 9, 0, 0},
    {0, 3, 7, 9, 0, 0},
    {3, 6, 7, 8, 0, 0},
    {4, 7, 8, 9, 0, 0},
    {3, 6, 8, 0, 0, 0},
    {1, 4, 4, 0, 0, 0},
    {0, 3, 3, 0, 0, 0},
    {3, 4, 8, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {5, 6, 6, 8, 0, 0},
    {0, 0, 5, 8, 0, 0},
    {2, 2, 5, 8, 0, 0},
    {5, 8, 8, 8, 0, 0},
    {3, 3, 5, 8, 0, 0},
    {5, 8, 0, 0, 0, 0},
    {1, 1, 5, 8, 0, 0},
};
constexpr int kSpecUpdProd[24][6] = {
    {0, 0, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
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
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0, d9 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z3), z1);
  b = __dmul_rn(__dmul_rn(c.kr(0), z4), z8);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(1), z9), z4);
  b = __dmul_rn(__dmul_rn(c.kr(1), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(2), z9), z3);
  b = __dmul_rn(__dmul_rn(c.kr(2), z8), z8);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d8 = __dadd_rn(d8, q);
  d8 = __dadd_rn(d8, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(3), z9), z3);
  b = __dmul_rn(__dmul_rn(c.kr(3), z6), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(4), z0), z4);
  b = __dmul_rn(__dmul_rn(c.kr(4), z3), z8);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z8), z8);
  b = __dmul_rn(__dmul_rn(c.kr(5), z6), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(6), z0), z8);
  b = __dmul_rn(__dmul_rn(c.kr(6), z6), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(7), z7), z1);
  b = __dmul_rn(__dmul_rn(c.kr(7), z9), z9);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z7), z8);
  b = __dmul_rn(__dmul_rn(c.kr(8), z6), z9);
  q = __dsub_rn(f, b);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(9), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(9), z9), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d7 = __dsub_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(10), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(10), z6), z8);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z7), z4);
  b = __dmul_rn(__dmul_rn(c.kr(11), z9), z8);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(c.kf(12), z6);
  b = __dmul_rn(__dmul_rn(c.kr(12), z3), z8);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d6 = __dsub_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(c.kf(13), z1);
  b = __dmul_rn(__dmul_rn(c.kr(13), z4), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(c.kf(14), z0);
  b = __dmul_rn(__dmul_rn(c.kr(14), z3), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z4), z3);
  b = __dmul_rn(c.kr(15), z8);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z3), z4);
  b = __dmul_rn(c.kr(16), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z5), z6);
  b = __dmul_rn(__dmul_rn(c.kr(17), z8), z6);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z5), z0);
  b = __dmul_rn(__dmul_rn(c.kr(18), z8), z0);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(19), z5), z2);
  b = __dmul_rn(__dmul_rn(c.kr(19), z8), z2);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z5), z8);
  b = __dmul_rn(__dmul_rn(c.kr(20), z8), z8);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d8 = __dsub_rn(d8, q);
  d8 = __dadd_rn(d8, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z5), z3);
  b = __dmul_rn(__dmul_rn(c.kr(21), z8), z3);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(c.kf(22), z5);
  b = __dmul_rn(c.kr(22), z8);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z5), z1);
  b = __dmul_rn(__dmul_rn(c.kr(23), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
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
}

constexpr int kFullN = 10, kFullR = 24;
constexpr int kFullLeft[24][3] = {
    {3, 1, -1},
    {9, 4, -1},
    {9, 3, -1},
    {9, 3, -1},
    {0, 4, -1},
    {8, 8, -1},
    {0, 8, -1},
    {7, 1, -1},
    {7, 8, -1},
    {7, 3, -1},
    {7, 3, -1},
    {7, 4, -1},
    {6, -1, -1},
    {1, -1, -1},
    {0, -1, -1},
    {4, 3, -1},
    {3, 4, -1},
    {5, 6, -1},
    {5, 0, -1},
    {5, 2, -1},
    {5, 8, -1},
    {5, 3, -1},
    {5, -1, -1},
    {5, 1, -1},
};
constexpr int kFullRight[24][3] = {
    {4, 8, -1},
    {8, 1, -1},
    {8, 8, -1},
    {6, 4, -1},
    {3, 8, -1},
    {6, 4, -1},
    {6, 3, -1},
    {9, 9, -1},
    {6, 9, -1},
    {9, 0, -1},
    {6, 8, -1},
    {9, 8, -1},
    {3, 8, -1},
    {4, 4, -1},
    {3, 3, -1},
    {8, -1, -1},
    {-1, 5, -1},
    {8, 6, -1},
    {8, 0, -1},
    {8, 2, -1},
    {8, 8, -1},
    {8, 3, -1},
    {8, -1, -1},
    {8, 1, -1},
};
constexpr int kFullNupd[24] = {4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 2, 4};
constexpr int kFullUpdK[24][6] = {
    {1, 3, 4, 8, 0, 0},
    {1, 4, 8, 9, 0, 0},
    {3, 8, 8, 9, 0, 0},
    {3, 4, 6, 9, 0, 0},
    {0, 3, 4, 8, 0, 0},
    {4, 6, 8, 8, 0, 0},
    {0, 3, 6, 8, 0, 0},
    {1, 7, 9, 9, 0, 0},
    {6, 7, 8, 9, 0, 0},
    {0, 3, 7, 9, 0, 0},
    {3, 6, 7, 8, 0, 0},
    {4, 7, 8, 9, 0, 0},
    {3, 6, 8, 0, 0, 0},
    {1, 4, 4, 0, 0, 0},
    {0, 3, 3, 0, 0, 0},
    {3, 4, 8, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {5, 6, 6, 8, 0, 0},
    {0, 0, 5, 8, 0, 0},
    {2, 2, 5, 8, 0, 0},
    {5, 8, 8, 8, 0, 0},
    {3, 3, 5, 8, 0, 0},
    {5, 8, 0, 0, 0, 0},
    {1, 1, 5, 8, 0, 0},
};
constexpr int kFullUpdProd[24][6] = {
    {0, 0, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
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
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0, d9 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z3), z1);
  b = __dmul_rn(__dmul_rn(c.kr(0), z4), z8);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(1), z9), z4);
  b = __dmul_rn(__dmul_rn(c.kr(1), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(2), z9), z3);
  b = __dmul_rn(__dmul_rn(c.kr(2), z8), z8);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d8 = __dadd_rn(d8, q);
  d8 = __dadd_rn(d8, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(3), z9), z3);
  b = __dmul_rn(__dmul_rn(c.kr(3), z6), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d9 = __dsub_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(4), z0), z4);
  b = __dmul_rn(__dmul_rn(c.kr(4), z3), z8);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z8), z8);
  b = __dmul_rn(__dmul_rn(c.kr(5), z6), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(6), z0), z8);
  b = __dmul_rn(__dmul_rn(c.kr(6), z6), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(7), z7), z1);
  b = __dmul_rn(__dmul_rn(c.kr(7), z9), z9);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d7 = __dsub_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z7), z8);
  b = __dmul_rn(__dmul_rn(c.kr(8), z6), z9);
  q = __dsub_rn(f, b);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(9), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(9), z9), z0);
  q = __dsub_rn(f, b);
  d0 = __dadd_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d7 = __dsub_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(10), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(10), z6), z8);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z7), z4);
  b = __dmul_rn(__dmul_rn(c.kr(11), z9), z8);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(c.kf(12), z6);
  b = __dmul_rn(__dmul_rn(c.kr(12), z3), z8);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d6 = __dsub_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(c.kf(13), z1);
  b = __dmul_rn(__dmul_rn(c.kr(13), z4), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(c.kf(14), z0);
  b = __dmul_rn(__dmul_rn(c.kr(14), z3), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z4), z3);
  b = __dmul_rn(c.kr(15), z8);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z3), z4);
  b = __dmul_rn(c.kr(16), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z5), z6);
  b = __dmul_rn(__dmul_rn(c.kr(17), z8), z6);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z5), z0);
  b = __dmul_rn(__dmul_rn(c.kr(18), z8), z0);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d0 = __dadd_rn(d0, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(19), z5), z2);
  b = __dmul_rn(__dmul_rn(c.kr(19), z8), z2);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d2 = __dadd_rn(d2, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z5), z8);
  b = __dmul_rn(__dmul_rn(c.kr(20), z8), z8);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d8 = __dsub_rn(d8, q);
  d8 = __dadd_rn(d8, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z5), z3);
  b = __dmul_rn(__dmul_rn(c.kr(21), z8), z3);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(c.kf(22), z5);
  b = __dmul_rn(c.kr(22), z8);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z5), z1);
  b = __dmul_rn(__dmul_rn(c.kr(23), z8), z1);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d8 = __dadd_rn(d8, q);
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
}

// Column J of I + factor * J: v[i] = A(i+1, J+1), each element's terms in
// reaction order.
template <int J, class S, typename LUT>
__device__ __forceinline__ void spec_column(const S& c, double factor, LUT (&v)[10]) {
  const double msf = -factor;
  double d;
  if constexpr (J == 0) {
    const double z4 = c.z(4), z5 = c.z(5), z8 = c.z(8), z9 = c.z(9);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(4), z4), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(6), z8), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(9), z9), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(c.kf(14), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z5), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(18), z8), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a0 = a0 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 1) {
    const double z3 = c.z(3), z5 = c.z(5), z7 = c.z(7), z8 = c.z(8);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z8), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(7), z7), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(c.kf(13), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(23), z5), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z8), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a1 = a1 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 2) {
    const double z5 = c.z(5), z8 = c.z(8);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(19), z5), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z8), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a2 = a2 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 3) {
    const double z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z9 = c.z(9);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(2), z9), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(3), z9), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(4), z8), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(6), z6), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(9), z7), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(10), z7), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z8), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z4), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(16), z4), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(21), z5), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z8), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a3 = a3 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 4) {
    const double z0 = c.z(0), z3 = c.z(3), z4 = c.z(4), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z9 = c.z(9);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(0), z8), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(1), z9), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z6), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(4), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(5), z6), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z7), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(16), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a4 = a4 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 5) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z6 = c.z(6), z8 = c.z(8);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(c.kr(16), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z6), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(19), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z8), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(21), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(c.kf(22), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(23), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a5 = a5 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 6) {
    const double z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z8 = c.z(8), z9 = c.z(9);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(3), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(5), z4), msf);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(6), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(8), z9), msf);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z8), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(c.kf(12), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z5), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z8), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a6 = a6 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 7) {
    const double z1 = c.z(1), z3 = c.z(3), z4 = c.z(4), z8 = c.z(8);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(7), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z8), factor);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(9), z3), factor);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(10), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a7 = a7 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 8) {
    const double z0 = c.z(0), z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z9 = c.z(9);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(0), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(2), z8), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(2), z8), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(4), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z8), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z8), factor);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(6), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z7), factor);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z6), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z9), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(c.kr(15), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z6), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(18), z0), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z2), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z5), factor);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z8), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z8), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z3), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(c.kr(22), msf);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z1), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = a8 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
  if constexpr (J == 9) {
    const double z0 = c.z(0), z3 = c.z(3), z4 = c.z(4), z6 = c.z(6), z8 = c.z(8), z9 = c.z(9);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(1), z4), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(2), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(3), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(7), z9), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(7), z9), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(8), z6), msf);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(9), z0), msf);
    a0 = (LUT)__dadd_rn((double)a0, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z8), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a9 = a9 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9;
  }
}

}  // namespace gen_tereza
}  // namespace nrg
