"""Generates mechanism-specialised right-hand sides and analytic iteration
matrices for the thread-per-cell integrator (nrg_b200/csrc/gen_*.cuh, one per
reference mechanism, and the index gen_mechanisms.cuh).

The table-driven kernels walk each reaction's reactant, product and update
lists through shared memory.  For the mechanism the library is built for, this
script writes the same arithmetic as straight-line code: the reacting
species' concentrations and the accumulators live in registers, and every
product and every update happens in the order of the table-driven loops, so
both paths give the same bits.  The tables of the specialised code are
emitted too; nrg_chem_create compares them with the parsed mechanism and uses
the specialised kernels only on an exact match.

    python nrg_b200/gen_mech.py            # the five reference decks, writes the headers

Needs a built libnrg_chem.so (it parses the decks with the library's own
reader, nrg_mech_tables).
"""
from __future__ import annotations

import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

# as kMergeUpTo in csrc/chem_device.cuh
MERGE_UP_TO = 16


def reduced_structure(t: dict, full: bool = False):
    """Reaction lists over the reacting species, built exactly as the host
    builds the device tables (build_dev_mech + reduce_dev_mech in capi.cu);
    full: over all species and reactions (build_dev_mech alone)."""
    N, R = t["n_species"], t["n_reactions"]
    co = t["coeffs"]
    left, right, upd = [], [], []
    for r in range(R):
        nl, nr = int(co[0][r][0]), int(co[1][r][0])
        raw_l = [int(co[0][r][1 + i]) for i in range(3)]
        raw_r = [int(co[1][r][1 + i]) for i in range(3)]
        left.append([(raw_l[i] - 1 if raw_l[i] != N + 1 else -1) if i < nl else -1 for i in range(3)])
        right.append([(raw_r[i] - 1 if raw_r[i] != N + 1 else -1) if i < nr else -1 for i in range(3)])
        u = []
        for k in range(1, N + 1):
            for i in range(nl):
                if raw_l[i] == k:
                    u.append((k - 1, 0))
            for i in range(nr):
                if raw_r[i] == k:
                    u.append((k - 1, 1))
        upd.append(u)
    if full:
        return N, R, left, right, upd
    reacts = sorted({s for r in range(R) for s in left[r] + right[r] if s >= 0})
    int_of = {k: i for i, k in enumerate(reacts)}
    left = [[int_of[s] if s >= 0 else -1 for s in row] for row in left]
    right = [[int_of[s] if s >= 0 else -1 for s in row] for row in right]
    upd = [[(int_of[k], p) for k, p in u] for u in upd]
    if len(reacts) <= MERGE_UP_TO:
        # reactions with equal lists are one reaction of the right-hand side
        # (their rate constants are added once per cell)
        first = [r for r in range(R) if (left[r], right[r]) not in list(zip(left[:r], right[:r]))]
        left, right, upd = ([x[r] for r in first] for x in (left, right, upd))
        R = len(first)
    return len(reacts), R, left, right, upd


def mul_chain(first: str, species) -> str:
    """first * z_a * z_b ... left to right, each product rounded on its own."""
    e = first
    for s in species:
        e = f"__dmul_rn({e}, z{s})"
    return e


def emit_tables_rhs(w, prefix: str, fn: str, N: int, R: int, left, right, upd) -> None:
    """The reaction lists and the right-hand side over N species and R reactions."""
    w(f"constexpr int {prefix}N = {N}, {prefix}R = {R};")

    def arr(nm, rows, width):
        w(f"constexpr int {nm}[{R}][{width}] = {{")
        for row in rows:
            w("    {" + ", ".join(str(x) for x in row) + "},")
        w("};")

    arr(f"{prefix}Left", left, 3)
    arr(f"{prefix}Right", right, 3)
    w(f"constexpr int {prefix}Nupd[{R}] = {{" + ", ".join(str(len(u)) for u in upd) + "};")
    arr(f"{prefix}UpdK", [[k for k, _ in u] + [0] * (6 - len(u)) for u in upd], 6)
    arr(f"{prefix}UpdProd", [[p for _, p in u] + [0] * (6 - len(u)) for u in upd], 6)
    w("")
    w("// zd = dC/dt at z (shared scratch in, shared scratch out)")
    w("template <class S>")
    w(f"__device__ __forceinline__ void {fn}(S& c) {{")
    used = {s for row in left + right for s in row if s >= 0}
    for k in range(N):
        if k in used:
            w(f"  const double z{k} = c.z({k});")
    w("  double " + ", ".join(f"d{k} = 0.0" for k in range(N)) + ";")
    w("  double f, b, q;")
    for r in range(R):
        w(f"  f = {mul_chain('c.kf(%d)' % r, [s for s in left[r] if s >= 0])};")
        w(f"  b = {mul_chain('c.kr(%d)' % r, [s for s in right[r] if s >= 0])};")
        w("  q = __dsub_rn(f, b);")
        for k, p in upd[r]:
            w(f"  d{k} = {'__dadd_rn' if p else '__dsub_rn'}(d{k}, q);")
    for k in range(N):
        w(f"  c.zd({k}) = d{k};")
    w("}")
    w("")


def emit(name: str, ns: str, reduced, full) -> str:
    NI, R, left, right, upd = reduced
    o = []
    w = o.append
    w(f"// Generated by nrg_b200/gen_mech.py from {name}.txt: do not edit.")
    w("// Straight-line right-hand side and analytic iteration matrix over the")
    w(f"// {NI} reacting species and {R} distinct reactions, and the right-hand side")
    w(f"// over all {full[0]} species and {full[1]} reactions; same operation order as the")
    w("// table-driven loops in chem_bdf.cuh, with the same explicitly rounded")
    w("// (never fused) operations.")
    w("#pragma once")
    w("")
    w("namespace nrg {")
    w(f"namespace {ns} {{")
    w("")
    emit_tables_rhs(w, "kSpec", "spec_rhs", NI, R, left, right, upd)
    emit_tables_rhs(w, "kFull", "full_rhs", *full)
    # analytic iteration matrix, column by column
    w("// Column J of I + factor * J: v[i] = A(i+1, J+1), each element's terms in")
    w("// reaction order.")
    w("template <int J, class S, typename LUT>")
    w(f"__device__ __forceinline__ void spec_column(const S& c, double factor, LUT (&v)[{NI}]) {{")
    w("  const double msf = -factor;")
    w("  double d;")
    for j in range(NI):
        names = set()
        body = []
        for r in range(R):
            for side in (0, 1):
                parts = right[r] if side else left[r]
                k = f"c.kr({r})" if side else f"c.kf({r})"
                for p in range(3):
                    if parts[p] != j:
                        continue
                    others = [parts[q] for q in range(3) if q != p and parts[q] >= 0]
                    names.update(others)
                    body.append(f"    d = __dmul_rn({mul_chain(k, others)}, {'msf' if side else 'factor'});")
                    for k2, pr in upd[r]:
                        body.append(f"    a{k2} = (LUT){'__dadd_rn' if pr else '__dsub_rn'}((double)a{k2}, d);")
        w(f"  if constexpr (J == {j}) {{")
        if names:
            w("    const double " + ", ".join(f"z{k} = c.z({k})" for k in sorted(names)) + ";")
        w("    LUT " + ", ".join(f"a{i} = (LUT)0" for i in range(NI)) + ";")
        o.extend(body)
        w(f"    a{j} = a{j} + 1;")
        w("    " + " ".join(f"v[{i}] = a{i};" for i in range(NI)))
        w("  }")
    w("}")
    w("")
    w(f"}}  // namespace {ns}")
    w("}  // namespace nrg")
    return "\n".join(o) + "\n"


def emit_index(names) -> str:
    """gen_mechanisms.cuh: the generated mechanisms, numbered from 1, and the
    host-side match of a parsed mechanism's tables against them: the reduced
    ones (the integrators that skip inert species) and the full ones (the
    reference mode) each on their own, for a deck that only lists an inert
    species elsewhere still has the reduced lists."""
    o = ["// Generated by nrg_b200/gen_mech.py: do not edit.",
         "// The mechanism-specialised codes, numbered from 1 (0 = table-driven).",
         "#pragma once", ""]
    o += [f'#include "gen_{n.lower()}.cuh"' for n in names]
    o += ["", "namespace nrg {", ""]
    o += [f"constexpr int kSpec{n.capitalize()} = {i + 1};" for i, n in enumerate(names)]
    o += ["", "template <int ID>", "struct SpecOf;"]
    for n in names:
        ns = f"gen_{n.lower()}"
        o += ["template <>", f"struct SpecOf<kSpec{n.capitalize()}> {{",
              f"  static constexpr int kN = {ns}::kSpecN, kR = {ns}::kSpecR;",
              f"  static constexpr int kFullN = {ns}::kFullN, kFullR = {ns}::kFullR;",
              "  template <class S>", f"  __device__ static void rhs(S& c) {{ {ns}::spec_rhs(c); }}",
              "  template <class S>", f"  __device__ static void rhs_full(S& c) {{ {ns}::full_rhs(c); }}",
              "  template <int J, class S, typename LUT>",
              f"  __device__ static void column(const S& c, double f, LUT (&v)[{ns}::kSpecN]) {{",
              f"    {ns}::spec_column<J>(c, f, v);", "  }", "};"]
    for fn, doc, count, species, prefix in (
            ("match_specialised_tables", "reduced", "m.RM", "m.NI", "kSpec"),
            ("match_specialised_full_tables", "full", "m.R", "m.N", "kFull")):
        o += ["", f"// 0 when the {doc} reaction lists match none of the generated codes.",
              "template <class M>", f"inline int {fn}(const M& m) {{"]
        for n in names:
            ns = f"gen_{n.lower()}"
            o += [f"  if ({species} == {ns}::{prefix}N && {count} == {ns}::{prefix}R) {{",
                  "    bool ok = true;",
                  f"    for (int r = 0; ok && r < {count}; ++r) {{",
                  f"      ok = m.nupd[r] == {ns}::{prefix}Nupd[r];",
                  "      for (int i = 0; ok && i < 3; ++i)",
                  f"        ok = m.left[r][i] == {ns}::{prefix}Left[r][i] && m.right[r][i] == {ns}::{prefix}Right[r][i];",
                  "      for (int u = 0; ok && u < m.nupd[r]; ++u)",
                  f"        ok = m.upd_k[r][u] == {ns}::{prefix}UpdK[r][u] && m.upd_prod[r][u] == {ns}::{prefix}UpdProd[r][u];",
                  "    }",
                  f"    if (ok) return kSpec{n.capitalize()};", "  }"]
        o += ["  return 0;", "}"]
    o += ["", "}  // namespace nrg", ""]
    return "\n".join(o)


def main() -> int:
    sys.path.insert(0, os.path.dirname(HERE))
    from nrg_b200 import ALL_MECHANISMS as MECHANISMS, mechanism_paths
    from nrg_b200.chemistry import mechanism_tables
    for name in MECHANISMS:
        t = mechanism_tables(*mechanism_paths(name))
        reduced, full = reduced_structure(t), reduced_structure(t, True)
        out = os.path.join(HERE, "csrc", f"gen_{name.lower()}.cuh")
        with open(out, "w") as fh:
            fh.write(emit(name, f"gen_{name.lower()}", reduced, full))
        print(f"wrote {out}: {reduced[0]} reacting species, {reduced[1]} distinct reactions")
    with open(os.path.join(HERE, "csrc", "gen_mechanisms.cuh"), "w") as fh:
        fh.write(emit_index(MECHANISMS))
    return 0


if __name__ == "__main__":
    sys.exit(main())
