// Generated by nrg_b200/gen_mech.py from ACETYLENE.txt: do not edit.
// Straight-line right-hand side and analytic iteration matrix over the
// 15 reacting species and 25 distinct reactions, and the right-hand side
// over all 17 species and 25 reactions; same operation order as the
// table-driven loops in chem_bdf.cuh, with the same explicitly rounded
// (never fused) operations.
#pragma once

namespace nrg {
namespace gen_acetylene {

constexpr int kSpecN = 15, kSpecR = 25;
constexpr int kSpecLeft[25][3] = {
    {3, 1, -1},
    {4, 2, -1},
    {4, 13, -1},
    {2, 5, -1},
    {4, 4, -1},
    {3, 1, -1},
    {12, 3, -1},
    {12, 3, -1},
    {12, 4, -1},
    {3, 4, -1},
    {5, -1, -1},
    {6, 4, -1},
    {7, 3, -1},
    {0, 1, -1},
    {0, 2, -1},
    {0, 4, -1},
    {9, 2, -1},
    {9, 3, -1},
    {10, 1, -1},
    {8, -1, -1},
    {8, 3, -1},
    {8, 4, -1},
    {11, -1, -1},
    {11, 3, -1},
    {14, 2, -1},
};
constexpr int kSpecRight[25][3] = {
    {4, 2, -1},
    {3, 1, -1},
    {5, 3, -1},
    {4, 4, -1},
    {2, 5, -1},
    {12, -1, -1},
    {4, 4, -1},
    {13, 1, -1},
    {5, 1, -1},
    {5, -1, -1},
    {3, 4, -1},
    {7, 3, -1},
    {6, 4, -1},
    {8, 6, -1},
    {10, 3, -1},
    {9, 3, -1},
    {10, 4, -1},
    {14, 6, -1},
    {6, 6, 4},
    {11, 3, -1},
    {11, 13, -1},
    {11, 5, -1},
    {6, 3, -1},
    {6, 13, -1},
    {8, 3, -1},
};
constexpr int kSpecNupd[25] = {4, 4, 4, 4, 4, 3, 4, 4, 4, 3, 3, 4, 4, 4, 4, 4, 4, 4, 5, 3, 4, 4, 3, 4, 4};
constexpr int kSpecUpdK[25][6] = {
    {1, 2, 3, 4, 0, 0},
    {1, 2, 3, 4, 0, 0},
    {3, 4, 5, 13, 0, 0},
    {2, 4, 4, 5, 0, 0},
    {2, 4, 4, 5, 0, 0},
    {1, 3, 12, 0, 0, 0},
    {3, 4, 4, 12, 0, 0},
    {1, 3, 12, 13, 0, 0},
    {1, 4, 5, 12, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {3, 4, 5, 0, 0, 0},
    {3, 4, 6, 7, 0, 0},
    {3, 4, 6, 7, 0, 0},
    {0, 1, 6, 8, 0, 0},
    {0, 2, 3, 10, 0, 0},
    {0, 3, 4, 9, 0, 0},
    {2, 4, 9, 10, 0, 0},
    {3, 6, 9, 14, 0, 0},
    {1, 4, 6, 6, 10, 0},
    {3, 8, 11, 0, 0, 0},
    {3, 8, 11, 13, 0, 0},
    {4, 5, 8, 11, 0, 0},
    {3, 6, 11, 0, 0, 0},
    {3, 6, 11, 13, 0, 0},
    {2, 3, 8, 14, 0, 0},
};
constexpr int kSpecUpdProd[25][6] = {
    {0, 1, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
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
  const double z13 = c.z(13);
  const double z14 = c.z(14);
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0, d9 = 0.0, d10 = 0.0, d11 = 0.0, d12 = 0.0, d13 = 0.0, d14 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z3), z1);
  b = __dmul_rn(__dmul_rn(c.kr(0), z4), z2);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d2 = __dadd_rn(d2, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(1), z4), z2);
  b = __dmul_rn(__dmul_rn(c.kr(1), z3), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d2 = __dsub_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  f = __dmul_rn(__dmul_rn(c.kf(2), z4), z13);
  b = __dmul_rn(__dmul_rn(c.kr(2), z5), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d13 = __dsub_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(3), z2), z5);
  b = __dmul_rn(__dmul_rn(c.kr(3), z4), z4);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(4), z4), z4);
  b = __dmul_rn(__dmul_rn(c.kr(4), z2), z5);
  q = __dsub_rn(f, b);
  d2 = __dadd_rn(d2, q);
  d4 = __dsub_rn(d4, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z3), z1);
  b = __dmul_rn(c.kr(5), z12);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(6), z12), z3);
  b = __dmul_rn(__dmul_rn(c.kr(6), z4), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d4 = __dadd_rn(d4, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(7), z12), z3);
  b = __dmul_rn(__dmul_rn(c.kr(7), z13), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d12 = __dsub_rn(d12, q);
  d13 = __dadd_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z12), z4);
  b = __dmul_rn(__dmul_rn(c.kr(8), z5), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(9), z3), z4);
  b = __dmul_rn(c.kr(9), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(c.kf(10), z5);
  b = __dmul_rn(__dmul_rn(c.kr(10), z3), z4);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z6), z4);
  b = __dmul_rn(__dmul_rn(c.kr(11), z7), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d6 = __dsub_rn(d6, q);
  d7 = __dadd_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(12), z7), z3);
  b = __dmul_rn(__dmul_rn(c.kr(12), z6), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d7 = __dsub_rn(d7, q);
  f = __dmul_rn(__dmul_rn(c.kf(13), z0), z1);
  b = __dmul_rn(__dmul_rn(c.kr(13), z8), z6);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d6 = __dadd_rn(d6, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(14), z0), z2);
  b = __dmul_rn(__dmul_rn(c.kr(14), z10), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d2 = __dsub_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d10 = __dadd_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z0), z4);
  b = __dmul_rn(__dmul_rn(c.kr(15), z9), z3);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z9), z2);
  b = __dmul_rn(__dmul_rn(c.kr(16), z10), z4);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d4 = __dadd_rn(d4, q);
  d9 = __dsub_rn(d9, q);
  d10 = __dadd_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z9), z3);
  b = __dmul_rn(__dmul_rn(c.kr(17), z14), z6);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d9 = __dsub_rn(d9, q);
  d14 = __dadd_rn(d14, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z10), z1);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(18), z6), z6), z4);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dadd_rn(d4, q);
  d6 = __dadd_rn(d6, q);
  d6 = __dadd_rn(d6, q);
  d10 = __dsub_rn(d10, q);
  f = __dmul_rn(c.kf(19), z8);
  b = __dmul_rn(__dmul_rn(c.kr(19), z11), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d8 = __dsub_rn(d8, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z8), z3);
  b = __dmul_rn(__dmul_rn(c.kr(20), z11), z13);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d8 = __dsub_rn(d8, q);
  d11 = __dadd_rn(d11, q);
  d13 = __dadd_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(21), z11), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d8 = __dsub_rn(d8, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(c.kf(22), z11);
  b = __dmul_rn(__dmul_rn(c.kr(22), z6), z3);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z11), z3);
  b = __dmul_rn(__dmul_rn(c.kr(23), z6), z13);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d6 = __dadd_rn(d6, q);
  d11 = __dsub_rn(d11, q);
  d13 = __dadd_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(24), z14), z2);
  b = __dmul_rn(__dmul_rn(c.kr(24), z8), z3);
  q = __dsub_rn(f, b);
  d2 = __dsub_rn(d2, q);
  d3 = __dadd_rn(d3, q);
  d8 = __dadd_rn(d8, q);
  d14 = __dsub_rn(d14, q);
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
  c.zd(13) = d13;
  c.zd(14) = d14;
}

constexpr int kFullN = 17, kFullR = 25;
constexpr int kFullLeft[25][3] = {
    {4, 1, -1},
    {5, 3, -1},
    {5, 14, -1},
    {3, 6, -1},
    {5, 5, -1},
    {4, 1, -1},
    {13, 4, -1},
    {13, 4, -1},
    {13, 5, -1},
    {4, 5, -1},
    {6, -1, -1},
    {7, 5, -1},
    {8, 4, -1},
    {0, 1, -1},
    {0, 3, -1},
    {0, 5, -1},
    {10, 3, -1},
    {10, 4, -1},
    {11, 1, -1},
    {9, -1, -1},
    {9, 4, -1},
    {9, 5, -1},
    {12, -1, -1},
    {12, 4, -1},
    {15, 3, -1},
};
constexpr int kFullRight[25][3] = {
    {5, 3, -1},
    {4, 1, -1},
    {6, 4, -1},
    {5, 5, -1},
    {3, 6, -1},
    {13, -1, -1},
    {5, 5, -1},
    {14, 1, -1},
    {6, 1, -1},
    {6, -1, -1},
    {4, 5, -1},
    {8, 4, -1},
    {7, 5, -1},
    {9, 7, -1},
    {11, 4, -1},
    {10, 4, -1},
    {11, 5, -1},
    {15, 7, -1},
    {7, 7, 5},
    {12, 4, -1},
    {12, 14, -1},
    {12, 6, -1},
    {7, 4, -1},
    {7, 14, -1},
    {9, 4, -1},
};
constexpr int kFullNupd[25] = {4, 4, 4, 4, 4, 3, 4, 4, 4, 3, 3, 4, 4, 4, 4, 4, 4, 4, 5, 3, 4, 4, 3, 4, 4};
constexpr int kFullUpdK[25][6] = {
    {1, 3, 4, 5, 0, 0},
    {1, 3, 4, 5, 0, 0},
    {4, 5, 6, 14, 0, 0},
    {3, 5, 5, 6, 0, 0},
    {3, 5, 5, 6, 0, 0},
    {1, 4, 13, 0, 0, 0},
    {4, 5, 5, 13, 0, 0},
    {1, 4, 13, 14, 0, 0},
    {1, 5, 6, 13, 0, 0},
    {4, 5, 6, 0, 0, 0},
    {4, 5, 6, 0, 0, 0},
    {4, 5, 7, 8, 0, 0},
    {4, 5, 7, 8, 0, 0},
    {0, 1, 7, 9, 0, 0},
    {0, 3, 4, 11, 0, 0},
    {0, 4, 5, 10, 0, 0},
    {3, 5, 10, 11, 0, 0},
    {4, 7, 10, 15, 0, 0},
    {1, 5, 7, 7, 11, 0},
    {4, 9, 12, 0, 0, 0},
    {4, 9, 12, 14, 0, 0},
    {5, 6, 9, 12, 0, 0},
    {4, 7, 12, 0, 0, 0},
    {4, 7, 12, 14, 0, 0},
    {3, 4, 9, 15, 0, 0},
};
constexpr int kFullUpdProd[25][6] = {
    {0, 1, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 1, 0, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {1, 0, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 1, 0, 0},
    {1, 0, 1, 0, 0, 0},
    {0, 0, 1, 1, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {1, 1, 0, 0, 0, 0},
    {0, 1, 0, 1, 0, 0},
    {0, 1, 1, 0, 0, 0},
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
  const double z9 = c.z(9);
  const double z10 = c.z(10);
  const double z11 = c.z(11);
  const double z12 = c.z(12);
  const double z13 = c.z(13);
  const double z14 = c.z(14);
  const double z15 = c.z(15);
  double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0, d4 = 0.0, d5 = 0.0, d6 = 0.0, d7 = 0.0, d8 = 0.0, d9 = 0.0, d10 = 0.0, d11 = 0.0, d12 = 0.0, d13 = 0.0, d14 = 0.0, d15 = 0.0, d16 = 0.0;
  double f, b, q;
  f = __dmul_rn(__dmul_rn(c.kf(0), z4), z1);
  b = __dmul_rn(__dmul_rn(c.kr(0), z5), z3);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d3 = __dadd_rn(d3, q);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(1), z5), z3);
  b = __dmul_rn(__dmul_rn(c.kr(1), z4), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  f = __dmul_rn(__dmul_rn(c.kf(2), z5), z14);
  b = __dmul_rn(__dmul_rn(c.kr(2), z6), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d14 = __dsub_rn(d14, q);
  f = __dmul_rn(__dmul_rn(c.kf(3), z3), z6);
  b = __dmul_rn(__dmul_rn(c.kr(3), z5), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(4), z5), z5);
  b = __dmul_rn(__dmul_rn(c.kr(4), z3), z6);
  q = __dsub_rn(f, b);
  d3 = __dadd_rn(d3, q);
  d5 = __dsub_rn(d5, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(5), z4), z1);
  b = __dmul_rn(c.kr(5), z13);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d13 = __dadd_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(6), z13), z4);
  b = __dmul_rn(__dmul_rn(c.kr(6), z5), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d5 = __dadd_rn(d5, q);
  d13 = __dsub_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(7), z13), z4);
  b = __dmul_rn(__dmul_rn(c.kr(7), z14), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d4 = __dsub_rn(d4, q);
  d13 = __dsub_rn(d13, q);
  d14 = __dadd_rn(d14, q);
  f = __dmul_rn(__dmul_rn(c.kf(8), z13), z5);
  b = __dmul_rn(__dmul_rn(c.kr(8), z6), z1);
  q = __dsub_rn(f, b);
  d1 = __dadd_rn(d1, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d13 = __dsub_rn(d13, q);
  f = __dmul_rn(__dmul_rn(c.kf(9), z4), z5);
  b = __dmul_rn(c.kr(9), z6);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  f = __dmul_rn(c.kf(10), z6);
  b = __dmul_rn(__dmul_rn(c.kr(10), z4), z5);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d6 = __dsub_rn(d6, q);
  f = __dmul_rn(__dmul_rn(c.kf(11), z7), z5);
  b = __dmul_rn(__dmul_rn(c.kr(11), z8), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d7 = __dsub_rn(d7, q);
  d8 = __dadd_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(12), z8), z4);
  b = __dmul_rn(__dmul_rn(c.kr(12), z7), z5);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d8 = __dsub_rn(d8, q);
  f = __dmul_rn(__dmul_rn(c.kf(13), z0), z1);
  b = __dmul_rn(__dmul_rn(c.kr(13), z9), z7);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d1 = __dsub_rn(d1, q);
  d7 = __dadd_rn(d7, q);
  d9 = __dadd_rn(d9, q);
  f = __dmul_rn(__dmul_rn(c.kf(14), z0), z3);
  b = __dmul_rn(__dmul_rn(c.kr(14), z11), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(15), z0), z5);
  b = __dmul_rn(__dmul_rn(c.kr(15), z10), z4);
  q = __dsub_rn(f, b);
  d0 = __dsub_rn(d0, q);
  d4 = __dadd_rn(d4, q);
  d5 = __dsub_rn(d5, q);
  d10 = __dadd_rn(d10, q);
  f = __dmul_rn(__dmul_rn(c.kf(16), z10), z3);
  b = __dmul_rn(__dmul_rn(c.kr(16), z11), z5);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d5 = __dadd_rn(d5, q);
  d10 = __dsub_rn(d10, q);
  d11 = __dadd_rn(d11, q);
  f = __dmul_rn(__dmul_rn(c.kf(17), z10), z4);
  b = __dmul_rn(__dmul_rn(c.kr(17), z15), z7);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d10 = __dsub_rn(d10, q);
  d15 = __dadd_rn(d15, q);
  f = __dmul_rn(__dmul_rn(c.kf(18), z11), z1);
  b = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(18), z7), z7), z5);
  q = __dsub_rn(f, b);
  d1 = __dsub_rn(d1, q);
  d5 = __dadd_rn(d5, q);
  d7 = __dadd_rn(d7, q);
  d7 = __dadd_rn(d7, q);
  d11 = __dsub_rn(d11, q);
  f = __dmul_rn(c.kf(19), z9);
  b = __dmul_rn(__dmul_rn(c.kr(19), z12), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(20), z9), z4);
  b = __dmul_rn(__dmul_rn(c.kr(20), z12), z14);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dadd_rn(d12, q);
  d14 = __dadd_rn(d14, q);
  f = __dmul_rn(__dmul_rn(c.kf(21), z9), z5);
  b = __dmul_rn(__dmul_rn(c.kr(21), z12), z6);
  q = __dsub_rn(f, b);
  d5 = __dsub_rn(d5, q);
  d6 = __dadd_rn(d6, q);
  d9 = __dsub_rn(d9, q);
  d12 = __dadd_rn(d12, q);
  f = __dmul_rn(c.kf(22), z12);
  b = __dmul_rn(__dmul_rn(c.kr(22), z7), z4);
  q = __dsub_rn(f, b);
  d4 = __dadd_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d12 = __dsub_rn(d12, q);
  f = __dmul_rn(__dmul_rn(c.kf(23), z12), z4);
  b = __dmul_rn(__dmul_rn(c.kr(23), z7), z14);
  q = __dsub_rn(f, b);
  d4 = __dsub_rn(d4, q);
  d7 = __dadd_rn(d7, q);
  d12 = __dsub_rn(d12, q);
  d14 = __dadd_rn(d14, q);
  f = __dmul_rn(__dmul_rn(c.kf(24), z15), z3);
  b = __dmul_rn(__dmul_rn(c.kr(24), z9), z4);
  q = __dsub_rn(f, b);
  d3 = __dsub_rn(d3, q);
  d4 = __dadd_rn(d4, q);
  d9 = __dadd_rn(d9, q);
  d15 = __dsub_rn(d15, q);
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
  c.zd(13) = d13;
  c.zd(14) = d14;
  c.zd(15) = d15;
  c.zd(16) = d16;
}

// Column J of I + factor * J: v[i] = A(i+1, J+1), each element's terms in
// reaction order.
template <int J, class S, typename LUT>
__device__ __forceinline__ void spec_column(const S& c, double factor, LUT (&v)[15]) {
  const double msf = -factor;
  double d;
  if constexpr (J == 0) {
    const double z1 = c.z(1), z2 = c.z(2), z4 = c.z(4);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(13), z1), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(14), z2), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z4), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    a0 = a0 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 1) {
    const double z0 = c.z(0), z3 = c.z(3), z5 = c.z(5), z10 = c.z(10), z13 = c.z(13);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z3), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z3), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(7), z13), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(8), z5), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(13), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z10), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a1 = a1 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 2) {
    const double z0 = c.z(0), z4 = c.z(4), z5 = c.z(5), z9 = c.z(9), z14 = c.z(14);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(0), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(1), z4), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(3), z5), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(4), z5), msf);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(14), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(16), z9), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(24), z14), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a14 = (LUT)__dsub_rn((double)a14, d);
    a2 = a2 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 3) {
    const double z1 = c.z(1), z4 = c.z(4), z5 = c.z(5), z6 = c.z(6), z7 = c.z(7), z8 = c.z(8), z9 = c.z(9), z10 = c.z(10), z11 = c.z(11), z12 = c.z(12);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(0), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(1), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kr(2), z5), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a13 = (LUT)__dsub_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kf(5), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(6), z12), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(7), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kf(9), z4), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z4), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(11), z7), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(12), z7), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(14), z10), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(15), z9), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z9), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a14 = (LUT)__dadd_rn((double)a14, d);
    d = __dmul_rn(__dmul_rn(c.kr(19), z11), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z8), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(22), z6), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(23), z11), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(24), z8), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a14 = (LUT)__dsub_rn((double)a14, d);
    a3 = a3 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 4) {
    const double z0 = c.z(0), z2 = c.z(2), z3 = c.z(3), z4 = c.z(4), z6 = c.z(6), z8 = c.z(8), z10 = c.z(10), z12 = c.z(12), z13 = c.z(13);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(0), z2), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(1), z2), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    d = __dmul_rn(__dmul_rn(c.kf(2), z13), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a13 = (LUT)__dsub_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z4), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(3), z4), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(4), z4), factor);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(4), z4), factor);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(6), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kr(6), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z12), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(9), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(10), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kf(11), z6), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z6), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(15), z0), factor);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kr(16), z10), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(18), z6), z6), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(21), z8), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a4 = a4 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 5) {
    const double z1 = c.z(1), z2 = c.z(2), z3 = c.z(3), z11 = c.z(11);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(2), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a13 = (LUT)__dsub_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kf(3), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(4), z2), msf);
    a2 = (LUT)__dadd_rn((double)a2, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(8), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(c.kr(9), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    d = __dmul_rn(c.kf(10), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a5 = (LUT)__dsub_rn((double)a5, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z11), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a5 = a5 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 6) {
    const double z3 = c.z(3), z4 = c.z(4), z6 = c.z(6), z8 = c.z(8), z13 = c.z(13), z14 = c.z(14);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(11), z4), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(12), z4), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kr(13), z8), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(__dmul_rn(c.kr(17), z14), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a14 = (LUT)__dadd_rn((double)a14, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(18), z6), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(__dmul_rn(c.kr(18), z6), z4), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(22), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z13), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    a6 = a6 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 7) {
    const double z3 = c.z(3);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(11), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a6 = (LUT)__dsub_rn((double)a6, d);
    a7 = (LUT)__dadd_rn((double)a7, d);
    d = __dmul_rn(__dmul_rn(c.kf(12), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a7 = (LUT)__dsub_rn((double)a7, d);
    a7 = a7 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 8) {
    const double z3 = c.z(3), z4 = c.z(4), z6 = c.z(6);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(13), z6), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    d = __dmul_rn(c.kf(19), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(20), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kf(21), z4), factor);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(24), z3), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a14 = (LUT)__dsub_rn((double)a14, d);
    a8 = a8 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 9) {
    const double z2 = c.z(2), z3 = c.z(3);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(15), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a9 = (LUT)__dadd_rn((double)a9, d);
    d = __dmul_rn(__dmul_rn(c.kf(16), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(17), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a14 = (LUT)__dadd_rn((double)a14, d);
    a9 = a9 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 10) {
    const double z1 = c.z(1), z3 = c.z(3), z4 = c.z(4);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(14), z3), msf);
    a0 = (LUT)__dsub_rn((double)a0, d);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kr(16), z4), msf);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a10 = (LUT)__dadd_rn((double)a10, d);
    d = __dmul_rn(__dmul_rn(c.kf(18), z1), factor);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a10 = (LUT)__dsub_rn((double)a10, d);
    a10 = a10 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 11) {
    const double z3 = c.z(3), z5 = c.z(5), z13 = c.z(13);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(19), z3), msf);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z13), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(21), z5), msf);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    d = __dmul_rn(c.kf(22), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    d = __dmul_rn(__dmul_rn(c.kf(23), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    a11 = a11 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 12) {
    const double z3 = c.z(3), z4 = c.z(4);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(c.kr(5), msf);
    a1 = (LUT)__dsub_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dadd_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(6), z3), factor);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a4 = (LUT)__dadd_rn((double)a4, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    d = __dmul_rn(__dmul_rn(c.kf(7), z3), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kf(8), z4), factor);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    a12 = a12 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 13) {
    const double z1 = c.z(1), z4 = c.z(4), z6 = c.z(6), z11 = c.z(11);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kf(2), z4), factor);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a4 = (LUT)__dsub_rn((double)a4, d);
    a5 = (LUT)__dadd_rn((double)a5, d);
    a13 = (LUT)__dsub_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(7), z1), msf);
    a1 = (LUT)__dadd_rn((double)a1, d);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a12 = (LUT)__dsub_rn((double)a12, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(20), z11), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a8 = (LUT)__dsub_rn((double)a8, d);
    a11 = (LUT)__dadd_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    d = __dmul_rn(__dmul_rn(c.kr(23), z6), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a11 = (LUT)__dsub_rn((double)a11, d);
    a13 = (LUT)__dadd_rn((double)a13, d);
    a13 = a13 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
  if constexpr (J == 14) {
    const double z2 = c.z(2), z6 = c.z(6);
    LUT a0 = (LUT)0, a1 = (LUT)0, a2 = (LUT)0, a3 = (LUT)0, a4 = (LUT)0, a5 = (LUT)0, a6 = (LUT)0, a7 = (LUT)0, a8 = (LUT)0, a9 = (LUT)0, a10 = (LUT)0, a11 = (LUT)0, a12 = (LUT)0, a13 = (LUT)0, a14 = (LUT)0;
    d = __dmul_rn(__dmul_rn(c.kr(17), z6), msf);
    a3 = (LUT)__dsub_rn((double)a3, d);
    a6 = (LUT)__dadd_rn((double)a6, d);
    a9 = (LUT)__dsub_rn((double)a9, d);
    a14 = (LUT)__dadd_rn((double)a14, d);
    d = __dmul_rn(__dmul_rn(c.kf(24), z2), factor);
    a2 = (LUT)__dsub_rn((double)a2, d);
    a3 = (LUT)__dadd_rn((double)a3, d);
    a8 = (LUT)__dadd_rn((double)a8, d);
    a14 = (LUT)__dsub_rn((double)a14, d);
    a14 = a14 + 1;
    v[0] = a0; v[1] = a1; v[2] = a2; v[3] = a3; v[4] = a4; v[5] = a5; v[6] = a6; v[7] = a7; v[8] = a8; v[9] = a9; v[10] = a10; v[11] = a11; v[12] = a12; v[13] = a13; v[14] = a14;
  }
}

}  // namespace gen_acetylene
}  // namespace nrg
