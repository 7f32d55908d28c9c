// Generated by nrg_b200/gen_mech.py: do not edit.
// The mechanism-specialised codes, numbered from 1 (0 = table-driven).
#pragma once

#include "gen_keromnes.cuh"
#include "gen_zhang.cuh"
#include "gen_tereza.cuh"
#include "gen_konnov.cuh"
#include "gen_acetylene.cuh"

namespace nrg {

constexpr int kSpecKeromnes = 1;
constexpr int kSpecZhang = 2;
constexpr int kSpecTereza = 3;
constexpr int kSpecKonnov = 4;
constexpr int kSpecAcetylene = 5;

template <int ID>
struct SpecOf;
template <>
struct SpecOf<kSpecKeromnes> {
  static constexpr int kN = gen_keromnes::kSpecN, kR = gen_keromnes::kSpecR;
  static constexpr int kFullN = gen_keromnes::kFullN, kFullR = gen_keromnes::kFullR;
  template <class S>
  __device__ static void rhs(S& c) { gen_keromnes::spec_rhs(c); }
  template <class S>
  __device__ static void rhs_full(S& c) { gen_keromnes::full_rhs(c); }
  template <int J, class S, typename LUT>
  __device__ static void column(const S& c, double f, LUT (&v)[gen_keromnes::kSpecN]) {
    gen_keromnes::spec_column<J>(c, f, v);
  }
};
template <>
struct SpecOf<kSpecZhang> {
  static constexpr int kN = gen_zhang::kSpecN, kR = gen_zhang::kSpecR;
  static constexpr int kFullN = gen_zhang::kFullN, kFullR = gen_zhang::kFullR;
  template <class S>
  __device__ static void rhs(S& c) { gen_zhang::spec_rhs(c); }
  template <class S>
  __device__ static void rhs_full(S& c) { gen_zhang::full_rhs(c); }
  template <int J, class S, typename LUT>
  __device__ static void column(const S& c, double f, LUT (&v)[gen_zhang::kSpecN]) {
    gen_zhang::spec_column<J>(c, f, v);
  }
};
template <>
struct SpecOf<kSpecTereza> {
  static constexpr int kN = gen_tereza::kSpecN, kR = gen_tereza::kSpecR;
  static constexpr int kFullN = gen_tereza::kFullN, kFullR = gen_tereza::kFullR;
  template <class S>
  __device__ static void rhs(S& c) { gen_tereza::spec_rhs(c); }
  template <class S>
  __device__ static void rhs_full(S& c) { gen_tereza::full_rhs(c); }
  template <int J, class S, typename LUT>
  __device__ static void column(const S& c, double f, LUT (&v)[gen_tereza::kSpecN]) {
    gen_tereza::spec_column<J>(c, f, v);
  }
};
template <>
struct SpecOf<kSpecKonnov> {
  static constexpr int kN = gen_konnov::kSpecN, kR = gen_konnov::kSpecR;
  static constexpr int kFullN = gen_konnov::kFullN, kFullR = gen_konnov::kFullR;
  template <class S>
  __device__ static void rhs(S& c) { gen_konnov::spec_rhs(c); }
  template <class S>
  __device__ static void rhs_full(S& c) { gen_konnov::full_rhs(c); }
  template <int J, class S, typename LUT>
  __device__ static void column(const S& c, double f, LUT (&v)[gen_konnov::kSpecN]) {
    gen_konnov::spec_column<J>(c, f, v);
  }
};
template <>
struct SpecOf<kSpecAcetylene> {
  static constexpr int kN = gen_acetylene::kSpecN, kR = gen_acetylene::kSpecR;
  static constexpr int kFullN = gen_acetylene::kFullN, kFullR = gen_acetylene::kFullR;
  template <class S>
  __device__ static void rhs(S& c) { gen_acetylene::spec_rhs(c); }
  template <class S>
  __device__ static void rhs_full(S& c) { gen_acetylene::full_rhs(c); }
  template <int J, class S, typename LUT>
  __device__ static void column(const S& c, double f, LUT (&v)[gen_acetylene::kSpecN]) {
    gen_acetylene::spec_column<J>(c, f, v);
  }
};

// 0 when the reduced reaction lists match none of the generated codes.
template <class M>
inline int match_specialised_tables(const M& m) {
  if (m.NI == gen_keromnes::kSpecN && m.RM == gen_keromnes::kSpecR) {
    bool ok = true;
    for (int r = 0; ok && r < m.RM; ++r) {
      ok = m.nupd[r] == gen_keromnes::kSpecNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_keromnes::kSpecLeft[r][i] && m.right[r][i] == gen_keromnes::kSpecRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_keromnes::kSpecUpdK[r][u] && m.upd_prod[r][u] == gen_keromnes::kSpecUpdProd[r][u];
    }
    if (ok) return kSpecKeromnes;
  }
  if (m.NI == gen_zhang::kSpecN && m.RM == gen_zhang::kSpecR) {
    bool ok = true;
    for (int r = 0; ok && r < m.RM; ++r) {
      ok = m.nupd[r] == gen_zhang::kSpecNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_zhang::kSpecLeft[r][i] && m.right[r][i] == gen_zhang::kSpecRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_zhang::kSpecUpdK[r][u] && m.upd_prod[r][u] == gen_zhang::kSpecUpdProd[r][u];
    }
    if (ok) return kSpecZhang;
  }
  if (m.NI == gen_tereza::kSpecN && m.RM == gen_tereza::kSpecR) {
    bool ok = true;
    for (int r = 0; ok && r < m.RM; ++r) {
      ok = m.nupd[r] == gen_tereza::kSpecNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_tereza::kSpecLeft[r][i] && m.right[r][i] == gen_tereza::kSpecRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_tereza::kSpecUpdK[r][u] && m.upd_prod[r][u] == gen_tereza::kSpecUpdProd[r][u];
    }
    if (ok) return kSpecTereza;
  }
  if (m.NI == gen_konnov::kSpecN && m.RM == gen_konnov::kSpecR) {
    bool ok = true;
    for (int r = 0; ok && r < m.RM; ++r) {
      ok = m.nupd[r] == gen_konnov::kSpecNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_konnov::kSpecLeft[r][i] && m.right[r][i] == gen_konnov::kSpecRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_konnov::kSpecUpdK[r][u] && m.upd_prod[r][u] == gen_konnov::kSpecUpdProd[r][u];
    }
    if (ok) return kSpecKonnov;
  }
  if (m.NI == gen_acetylene::kSpecN && m.RM == gen_acetylene::kSpecR) {
    bool ok = true;
    for (int r = 0; ok && r < m.RM; ++r) {
      ok = m.nupd[r] == gen_acetylene::kSpecNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_acetylene::kSpecLeft[r][i] && m.right[r][i] == gen_acetylene::kSpecRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_acetylene::kSpecUpdK[r][u] && m.upd_prod[r][u] == gen_acetylene::kSpecUpdProd[r][u];
    }
    if (ok) return kSpecAcetylene;
  }
  return 0;
}

// 0 when the full reaction lists match none of the generated codes.
template <class M>
inline int match_specialised_full_tables(const M& m) {
  if (m.N == gen_keromnes::kFullN && m.R == gen_keromnes::kFullR) {
    bool ok = true;
    for (int r = 0; ok && r < m.R; ++r) {
      ok = m.nupd[r] == gen_keromnes::kFullNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_keromnes::kFullLeft[r][i] && m.right[r][i] == gen_keromnes::kFullRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_keromnes::kFullUpdK[r][u] && m.upd_prod[r][u] == gen_keromnes::kFullUpdProd[r][u];
    }
    if (ok) return kSpecKeromnes;
  }
  if (m.N == gen_zhang::kFullN && m.R == gen_zhang::kFullR) {
    bool ok = true;
    for (int r = 0; ok && r < m.R; ++r) {
      ok = m.nupd[r] == gen_zhang::kFullNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_zhang::kFullLeft[r][i] && m.right[r][i] == gen_zhang::kFullRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_zhang::kFullUpdK[r][u] && m.upd_prod[r][u] == gen_zhang::kFullUpdProd[r][u];
    }
    if (ok) return kSpecZhang;
  }
  if (m.N == gen_tereza::kFullN && m.R == gen_tereza::kFullR) {
    bool ok = true;
    for (int r = 0; ok && r < m.R; ++r) {
      ok = m.nupd[r] == gen_tereza::kFullNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_tereza::kFullLeft[r][i] && m.right[r][i] == gen_tereza::kFullRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_tereza::kFullUpdK[r][u] && m.upd_prod[r][u] == gen_tereza::kFullUpdProd[r][u];
    }
    if (ok) return kSpecTereza;
  }
  if (m.N == gen_konnov::kFullN && m.R == gen_konnov::kFullR) {
    bool ok = true;
    for (int r = 0; ok && r < m.R; ++r) {
      ok = m.nupd[r] == gen_konnov::kFullNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_konnov::kFullLeft[r][i] && m.right[r][i] == gen_konnov::kFullRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_konnov::kFullUpdK[r][u] && m.upd_prod[r][u] == gen_konnov::kFullUpdProd[r][u];
    }
    if (ok) return kSpecKonnov;
  }
  if (m.N == gen_acetylene::kFullN && m.R == gen_acetylene::kFullR) {
    bool ok = true;
    for (int r = 0; ok && r < m.R; ++r) {
      ok = m.nupd[r] == gen_acetylene::kFullNupd[r];
      for (int i = 0; ok && i < 3; ++i)
        ok = m.left[r][i] == gen_acetylene::kFullLeft[r][i] && m.right[r][i] == gen_acetylene::kFullRight[r][i];
      for (int u = 0; ok && u < m.nupd[r]; ++u)
        ok = m.upd_k[r][u] == gen_acetylene::kFullUpdK[r][u] && m.upd_prod[r][u] == gen_acetylene::kFullUpdProd[r][u];
    }
    if (ok) return kSpecAcetylene;
  }
  return 0;
}

}  // namespace nrg
