"""Mechanism-specific CUDA code for the right-hand side (like CEPTR does for
the reference's mechanisms).

For a flattened mechanism this writes a device function

    void gen_rhs_<name>(const double* y, const double* F, double* out, ...)

with every rate constant, stoichiometric coefficient, efficiency and NASA-7
coefficient as an operand in constant memory, so that concentrations and production rates live
in registers and no table is read.  The formulas are the ones of the
table-driven right-hand side (Chemkin formalism: Arrhenius, third body,
Lindemann / Troe falloff, reverse rates from Kc); Kc is formed from one
exponential per species instead of one per reaction.

The function is selected at handle creation by a 64-bit FNV-1a digest of the
mechanism description (mechanism_digest), computed identically here and in
the library.
"""
from __future__ import annotations

import numpy as np

FNV_OFFSET = 0xcbf29ce484222325
FNV_PRIME = 0x100000001b3


def _fnv(h: int, data: bytes) -> int:
    for b in data:
        h ^= b
        h = (h * FNV_PRIME) & 0xFFFFFFFFFFFFFFFF
    return h


def mechanism_digest(flat) -> int:
    """FNV-1a over the description arrays in b200chem_mech_desc order."""
    a = flat.arrays
    h = FNV_OFFSET
    h = _fnv(h, np.array([flat.n_species, flat.n_reactions, flat.n_eff], np.int32).tobytes())
    for key, dt in (("mw", np.float64), ("nasa", np.float64), ("rtype", np.int32), ("rflags", np.int32),
                    ("arr", np.float64), ("arr_lo", np.float64), ("arr_rev", np.float64), ("troe", np.float64),
                    ("sp", np.int32), ("nu", np.int32), ("eff_ptr", np.int32)):
        h = _fnv(h, np.ascontiguousarray(a[key], dt).tobytes())
    ne = flat.n_eff
    h = _fnv(h, np.ascontiguousarray(a["eff_sp"][:ne], np.int32).tobytes())
    h = _fnv(h, np.ascontiguousarray(a["eff_val"][:ne], np.float64).tobytes())
    return h


def _d(x: float) -> str:
    return repr(float(x))


KRU = 8.31446261815324e7  # erg/mol/K, as in the device code
PATM = 1013250.0  # dyn/cm^2
# largest magnitude of an exponential's argument in the generated code (its
# exponential has no overflow or underflow handling)
EXP_LIMIT = 690.0


def _nasa_g(nasa, T):
    """g/RT of every species at T (numpy, NASA-7)."""
    a = np.where((T < nasa[:, :1]), nasa[:, 1:8], nasa[:, 8:15]).T
    h = a[0] + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5))) + a[5] / T
    return h - (a[0] * np.log(T) + T * (a[1] + T * (a[2] / 2 + T * (a[3] / 3 + T * a[4] / 4))) + a[6])


def temperature_range(flat) -> tuple:
    """Widest range of temperatures around 1000 K in which every exponential of
    the generated right-hand side (Troe's may underflow, not overflow) and every
    product of species exponentials, after each of its factors, stay within
    EXP_LIMIT; outside it the table form is used."""
    a = flat.arrays
    nu, sp = a["nu"], a["sp"]

    def fine(T):
        g = _nasa_g(a["nasa"], T)
        ok = np.abs(g).max() <= EXP_LIMIT
        lnu = np.log(T * KRU / PATM)
        for j in range(flat.n_reactions):
            for key in ("arr", "arr_lo", "arr_rev"):
                ok &= abs(a[key][j][0] + a[key][j][1] * np.log(T) - a[key][j][2] / T) <= EXP_LIMIT
            if a["rtype"][j] == 3:
                _, t3, t1, t2 = a["troe"][j]
                ok &= max(-T / t3, -T / t1, -t2 / T if a["rflags"][j] & 4 else 0.0) <= EXP_LIMIT
            # exponents of the factors in the order of the product: products,
            # reactants, powers of the standard concentration
            sides = [[sp[j, s] for s in r if sp[j, s] >= 0 for _ in range(int(nu[j, s]))] for r in (range(4), range(4, 8))]
            dn = len(sides[1]) - len(sides[0])
            e = np.concatenate([g[sides[1]], -g[sides[0]], np.full(abs(dn), np.sign(dn) * lnu)])
            ok &= np.abs(np.cumsum(e)).max() <= EXP_LIMIT
        return bool(ok)

    lo, hi = 1000.0, 1000.0
    while lo > 50.0 and fine(lo - 5.0):
        lo -= 5.0
    while hi < 20000.0 and fine(hi + 50.0):
        hi += 50.0
    return lo, hi


def _chain(factors) -> str:
    """Left-to-right product, each multiply rounded on its own."""
    out = factors[0]
    for f in factors[1:]:
        out = f"__dmul_rn({out}, {f})"
    return out


def generate(flat, name: str) -> str:
    """The right-hand side of one mechanism, one thread per cell.  Every
    operation is written with its rounding (fma, __dmul_rn, ...) and in the
    order of the table-driven warp form (rhs_warp in react_rhs.cu), so that
    both give the same bits.  sE, sI: exp(g/RT) and exp(-g/RT) of the species,
    per-thread columns of shared memory (stride ss): they would take the
    registers that the concentrations and rates need.  Exponentials are
    evaluated four at a time, in the order the reactions need them."""
    a = flat.arrays
    N, R = flat.n_species, flat.n_reactions
    mw = a["mw"]
    nasa = a["nasa"]  # [N][15]
    if not np.all(nasa[:, 0] == nasa[0, 0]):
        raise ValueError("generated right-hand side needs one common NASA-7 midpoint temperature")
    tlo, thi = temperature_range(flat)
    out, consts = [], {}
    w = out.append

    def _d(v):
        """A coefficient: an entry of the mechanism's constant-memory array, which
        the FP64 instructions take as an operand (a literal takes two moves)."""
        v = float(v)
        if v in (0.0, 1.0, -1.0, 2.0, -2.0):
            return repr(v)
        return f"kc_{name}[{consts.setdefault(v, len(consts))}]"

    head = [f"// mechanism {name}: {N} species, {R} reactions",
            f"constexpr unsigned long long kGenDigest_{name} = {mechanism_digest(flat)}ull;",
            f"constexpr double kGenTlo_{name} = {tlo!r}, kGenThi_{name} = {thi!r};", "#ifdef B200_GEN_FUNCTIONS"]
    w(f"__device__ __forceinline__ void gen_rhs_{name}(const double* __restrict__ y, "
      f"const double* __restrict__ F, double* __restrict__ out, double* __restrict__ sE, double* __restrict__ sI, "
      f"int ss) {{")
    w(f"  const double T = y[{N}];")
    w("  const double lnT = log(T), invT = 1.0 / T;")
    w("  const double u = __dmul_rn(T, kRu / kPatm), iu = 1.0 / u;")
    w("  const double oml = 1.0 - lnT;")
    w(f"  const bool lo = T < {float(nasa[0, 0])!r};")
    w(f"  double C[{N}], wd[{N}];")
    w("  double Ctot = 0.0, rcp = 0.0;")
    for k0 in range(0, N, 2):
        ks = range(k0, min(N, k0 + 2))
        w("  { double x[4] = {0.0, 0.0, 0.0, 0.0};")
        for b, cond in (("lo", 1), ("hi", 8)):
            w("    if (lo) {" if b == "lo" else "    } else {")
            for k in ks:
                c = nasa[k, cond:cond + 7]
                cg = [c[0], c[1] / -2.0, c[2] / -6.0, c[3] / -12.0, c[4] / -20.0, c[5], c[6]]
                w(f"      x[{2 * (k - k0)}] = nasa_g({', '.join(_d(v) for v in cg)}, T, invT, oml);")
                w(f"      x[{2 * (k - k0) + 1}] = nasa_cp({', '.join(_d(v) for v in c[:5])}, T);")
        w("    }")
        for k in ks:
            i = 2 * (k - k0)
            w(f"    C[{k}] = __dmul_rn(y[{k}], {_d(1.0 / mw[k])}); wd[{k}] = 0.0; Ctot = __dadd_rn(Ctot, C[{k}]);")
            w(f"    rcp = fma(C[{k}], x[{i + 1}], rcp); x[{i + 1}] = -x[{i}];")
        w("    const Exp4 v = pexp4(x[0], x[1], x[2], x[3]);")
        for k in ks:
            i = 2 * (k - k0)
            w(f"    sE[{k} * ss] = v.x[{i}]; sI[{k} * ss] = v.x[{i + 1}];")
        w("  }")
    sp, nu = a["sp"], a["nu"]
    effp, effs, effv = a["eff_ptr"], a["eff_sp"], a["eff_val"]

    def arrh(c):
        t = _d(c[0])
        if c[1] != 0.0:
            t = f"fma({_d(c[1])}, lnT, {t})"
        if c[2] != 0.0:
            t = f"fma({_d(-c[2])}, invT, {t})"
        return t

    # arguments of every exponential in reaction order
    args, where, last = [], {}, {}
    for j in range(R):
        typ, fl = int(a["rtype"][j]), int(a["rflags"][j])
        where[j] = len(args)
        args.append(arrh(a["arr"][j]))
        if typ >= 2:
            args.append(arrh(a["arr_lo"][j]))
        if typ == 3:
            _, t3, t1, t2 = a["troe"][j]
            args += [f"fexp_arg(__dmul_rn(-T, {_d(1.0 / t3)}))", f"fexp_arg(__dmul_rn(-T, {_d(1.0 / t1)}))"]
            if fl & 4:
                args.append(f"fexp_arg(__dmul_rn({_d(-t2)}, invT))")
        if fl & 2:
            where[(j, "rev")] = len(args)
            args.append(arrh(a["arr_rev"][j]))
        last[j] = len(args)
    done = 0

    def x(i):
        return f"x{i // 4}.x[{i % 4}]"

    for j in range(R):
        while done < last[j]:
            four = (args[done:done + 4] + ["0.0"] * 4)[:4]
            w(f"  const Exp4 x{done // 4} = pexp4({', '.join(four)});")
            done += 4
        typ, fl = int(a["rtype"][j]), int(a["rflags"][j])
        i = where[j]
        w(f"    {{ // reaction {j}")
        if typ != 0:
            m = "Ctot"
            for q in range(effp[j], effp[j + 1]):
                e = effv[q] - 1.0
                if e != 0.0:
                    m = f"fma({_d(e)}, C[{int(effs[q])}], {m})"
            w(f"      const double M = {m};")
        if typ == 2:
            w(f"      const double kf = lindemann({x(i)}, {x(i + 1)}, M);")
        elif typ == 3:
            al = float(a["troe"][j][0])
            fc = f"fma({_d(1.0 - al)}, {x(i + 2)}, __dmul_rn({_d(al)}, {x(i + 3)}))"
            if fl & 4:
                fc = f"__dadd_rn({fc}, {x(i + 4)})"
            w(f"      const double kf = troe({x(i)}, {x(i + 1)}, M, {fc});")
        else:
            w(f"      const double kf = {x(i)};")
        sides = [[int(sp[j, s]) for s in r if sp[j, s] >= 0 for _ in range(int(nu[j, s]))]
                 for r in (range(4), range(4, 8))]
        prods = [_chain([f"C[{k}]" for k in sd]) if sd else "1.0" for sd in sides]
        if fl & 2:
            w(f"      double q = __dsub_rn(__dmul_rn(kf, {prods[0]}), __dmul_rn({x(where[(j, 'rev')])}, {prods[1]}));")
        elif fl & 1:
            sdn = len(sides[1]) - len(sides[0])
            fac = [f"sE[{k} * ss]" for k in sides[1]] + [f"sI[{k} * ss]" for k in sides[0]]
            fac += ["u"] * sdn if sdn > 0 else ["iu"] * -sdn
            w(f"      double q = __dmul_rn(kf, fma(-{_chain(fac)}, {prods[1]}, {prods[0]}));")
        else:
            w(f"      double q = __dmul_rn(kf, {prods[0]});")
        if typ == 1:
            w("      q = __dmul_rn(q, M);")
        net = {}
        for sgn, sd in zip((-1, 1), sides):
            for k in sd:
                net[k] = net.get(k, 0) + sgn
        for k, v in sorted(net.items()):
            if v:
                w(f"      wd[{k}] = fma({_d(v)}, q, wd[{k}]);")
        w("    }")
    w("  double hs = 0.0;")
    for k in range(N):
        w("  { double hRT;")
        for b, cond in (("lo", 1), ("hi", 8)):
            c = nasa[k, cond:cond + 7]
            ch = [c[0], c[1] / 2.0, c[2] / 3.0, c[3] / 4.0, c[4] / 5.0, c[5]]
            w(f"    {'if (lo)' if b == 'lo' else 'else'} hRT = nasa_h({', '.join(_d(v) for v in ch)}, T, invT);")
        w(f"    const double yd = fma(wd[{k}], {_d(mw[k])}, F[{k}]);")
        w(f"    out[{k}] = yd; hs = fma(__dmul_rn(hRT, {_d(KRU / mw[k])}), yd, hs); }}")
    w(f"  out[{N}] = fma(-T, hs, F[{N}]) / __dmul_rn(kRu, rcp);")
    w("}")
    w("#endif")
    vals = [repr(v) for v in consts]
    head.append(f"static __constant__ double kc_{name}[{len(vals)}] = {{")
    head += ["  " + ", ".join(vals[i:i + 6]) + "," for i in range(0, len(vals), 6)] + ["};"]
    return "\n".join(head + out) + "\n"


def generate_bundled() -> str:
    """Header with the generated right-hand sides of the bundled mechanisms: their
    digests and temperature ranges, and the functions where B200_GEN_FUNCTIONS is
    defined."""
    from . import mechanism as mechmod
    parts = ["// gen_mechs.cuh -- generated by pelelmex_b200.mechgen; do not edit.",
             "#pragma once", "#include \"rate_math.cuh\"", "namespace b200 {", "namespace gen {"]
    for name in ("synth_h2_9", "synth_ch4_21", "synth_c12_53"):
        flat = mechmod.flatten(mechmod.builtin(name))
        parts.append(generate(flat, name))
    parts += ["}  // namespace gen", "}  // namespace b200"]
    return "\n".join(parts) + "\n"


def _c_array(ctype: str, name: str, values, per_line: int = 6) -> str:
    vals = [repr(float(v)) if ctype == "double" else str(int(v)) for v in np.ravel(values)]
    if not vals:
        vals = ["0"]
    lines = [", ".join(vals[i:i + per_line]) for i in range(0, len(vals), per_line)]
    return f"static const {ctype} {name}[{len(vals)}] = {{\n  " + ",\n  ".join(lines) + "\n};\n"


def generate_mech_desc(flat, name: str) -> str:
    """C++ translation unit defining b200chem_make_mech_desc() for one
    mechanism: the flat description (the data a CEPTR-generated mechanism
    bakes into code) as static tables, so a PelePhysics build links the
    ReactorB200 shim without hand-written mechanism code.  The digest it
    carries in a comment is the one the library computes for it."""
    a = flat.arrays
    ne = flat.n_eff
    out = [f"// b200chem mechanism description of {name}: {flat.n_species} species, {flat.n_reactions} "
           f"reactions.", "// Generated by pelelmex_b200.mechgen; do not edit.",
           f"// digest 0x{mechanism_digest(flat):016x}", '#include "b200chem.h"', "", "namespace {"]
    for key, ct in (("mw", "double"), ("nasa", "double"), ("rtype", "int32_t"), ("rflags", "int32_t"),
                    ("arr", "double"), ("arr_lo", "double"), ("arr_rev", "double"), ("troe", "double"),
                    ("sp", "int32_t"), ("nu", "int32_t"), ("eff_ptr", "int32_t")):
        out.append(_c_array(ct, f"k_{key}", a[key]))
    out.append(_c_array("int32_t", "k_eff_sp", a["eff_sp"][:max(ne, 0)]))
    out.append(_c_array("double", "k_eff_val", a["eff_val"][:max(ne, 0)]))
    out += ["}  // namespace", "", "b200chem_mech_desc b200chem_make_mech_desc() {", "  b200chem_mech_desc d{};",
            f"  d.n_species = {flat.n_species};", f"  d.n_reactions = {flat.n_reactions};", f"  d.n_eff = {ne};"]
    for key in ("mw", "nasa", "rtype", "rflags", "arr", "arr_lo", "arr_rev", "troe", "sp", "nu", "eff_ptr",
                "eff_sp", "eff_val"):
        out.append(f"  d.{key} = k_{key};")
    out += ["  return d;", "}", ""]
    return "\n".join(out)


def main(argv=None):
    """python -m pelelmex_b200.mechgen --mech-desc MECHANISM --out FILE.cpp

    MECHANISM is a bundled mechanism name or a Cantera-style YAML file."""
    import argparse
    from pathlib import Path
    from . import mechanism as mechmod
    p = argparse.ArgumentParser()
    p.add_argument("--mech-desc", required=True)
    p.add_argument("--out", required=True)
    a = p.parse_args(argv)
    src = a.mech_desc
    mech = mechmod.load(src) if Path(src).exists() else mechmod.builtin(src)
    Path(a.out).write_text(generate_mech_desc(mechmod.flatten(mech), mech.name if hasattr(mech, "name") else src))


if __name__ == "__main__":
    main()
