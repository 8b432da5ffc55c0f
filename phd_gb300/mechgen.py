"""Mechanism compiler: the constant-volume reactor right-hand side of one
CHEMKIN mechanism as CUDA code of its own.

The chemistry kernels evaluate CHEMKIN's rate expressions (CKCVBS, CKHMS,
CKRATT, CKRATX, CKWYR; chemkin/vode.f) for whatever mechanism the caller
uploads, walking its reaction tables at run time.  Species concentrations,
rates of progress and production rates are then indexed by table entries,
so they live in local memory, and every term costs a table load and a
branch.  For a mechanism known when the library is built this module writes
the same expressions, in the same operation order, for its reactions alone:
in the composition part the reaction loops are unrolled, indices fixed, absent
terms dropped and the table entries literals; the Arrhenius and NASA terms of
the temperature part stay loops, over constant tables, since unrolled they
push the integrator out of the instruction cache.
The arithmetic is the generic form's (fun_tpart / fun_cpart in chem.cu),
operation for operation, so a host build of the two gives identical bits.

Supported: irreversible reactions, reverse rates from the equilibrium
constant (CKSMH's entropy-enthalpy difference) or from explicit parameters
(REV), +M third bodies with efficiencies, Lindemann, SRI and Troe (3 or 4
parameter) fall-off with the (+M) collider or one species (+K), and
Landau-Teller factors on forward (LT) and explicit reverse (RLT) rates.

``python -m phd_gb300.mechgen`` rewrites ``csrc/chem_gen.cuh`` from the
shipped mechanism; a test checks that the committed file is what this
module writes.
"""
import os
import struct

HERE = os.path.dirname(os.path.abspath(__file__))
LT_P1 = 1.0 / 3.0        # the Landau-Teller exponents of chem.cu (kLtP1, kLtP2)
LT_P2 = 2.0 * LT_P1
OUT = os.path.join(HERE, "csrc", "chem_gen.cuh")


def lit(x):
    """A double literal that reads back to exactly x (C99/C++17 hex float)."""
    x = float(x)
    if x == 0.0:
        return "-0.0" if struct.pack(">d", x)[0] & 0x80 else "0.0"
    return "(%s)" % x.hex() if x < 0 else x.hex()


def bits(x):
    return "0x%016xULL" % struct.unpack("<Q", struct.pack("<d", float(x)))[0]


def powi_expr(x, m):
    """powi(x, m) of chem.cu for m > 0, unrolled: the same products in the
    same order (y = 1.0 * x^2 is x^2 exactly)."""
    assert m > 0
    n = m
    y = x if n % 2 else None
    xx = x
    n >>= 1
    while n:
        xx = "(%s * %s)" % (xx, xx)
        if n % 2:
            y = xx if y is None else "(%s * %s)" % (y, xx)
        n >>= 1
    return y


def _reactions(m):
    out = []
    for i in range(m.ii):
        r = {"i": i, "nuk": list(m.nuk[i]), "nu": list(m.nu[i]), "par": list(m.par[i]), "rev": m.rev[i],
             "rpar": list(m.rpar[i]), "thb": m.thb[i], "fall": m.fall[i], "low": list(m.low[i]),
             "troe": list(m.troe[i]), "sri": list(m.sri[i]), "kfal": m.kfal[i],
             "lt": list(m.lt[i]), "rlt": list(m.rlt[i]),
             "eff": [m.eff[i][k] for k in range(m.kk)]}
        if r["fall"] not in (0, 1, 2, 3, 4):
            raise NotImplementedError("reaction %d: fall-off form %d" % (i, r["fall"]))
        if r["nu"][0] == 0:
            raise NotImplementedError("reaction %d: no reactant" % i)
        out.append(r)
    return out


def generate(m, name="h2air9", source="phd_gb300/data/h2_sandiego12.inp"):
    kk = m.kk
    R = _reactions(m)
    rev = [r["i"] for r in R if r["rev"] != 0]
    eqk = any(r["rev"] == 1 for r in R)
    fall = [r["i"] for r in R if r["fall"]]
    troe = [r["i"] for r in R if r["fall"] > 1]
    tr_slot = {i: q for q, i in enumerate(troe)}
    wt_inv = [1.0 / m.wt[k] for k in range(kk)]
    ru_wt = [m.ru / m.wt[k] for k in range(kk)]

    # the Arrhenius expressions A exp(b ln T - E/R / T) in one table: forward,
    # explicit reverse and low-pressure rate constants
    arr = [r["par"] for r in R]
    kr_at, lo_at = {}, {}
    for r in R:
        if r["rev"] == 2:
            kr_at[r["i"]] = len(arr)
            arr.append(r["rpar"])
    for r in R:
        if r["rev"] == 1:   # from the equilibrium constant: a slot without an expression
            kr_at[r["i"]] = None
    for r in R:
        if r["fall"]:
            lo_at[r["i"]] = len(arr)
            arr.append(r["low"])
    n_exp = len(arr)
    for i in [i for i in kr_at if kr_at[i] is None]:
        kr_at[i] = len(arr)
        arr.append(None)
    L = []
    w = L.append
    w("// Generated by phd_gb300/mechgen.py from %s -- do not edit." % source)
    w("// The constant-volume reactor right-hand side of this mechanism (%d species," % kk)
    w("// %d reactions): the expressions and operation order of fun_tpart / fun_cpart" % m.ii)
    w("// in chem.cu, the composition part straight-line code with the mechanism's numbers")
    w("// as literals, the Arrhenius and NASA terms loops over constant tables.")
    w("#pragma once")
    w("")
    w("namespace chem_gen {")
    w("")
    w("constexpr int KK = %d;" % kk)
    w("")
    w("// temperature terms of one right-hand side; the finite-difference Jacobian's")
    w("// species columns reuse them (rc_drive)")
    w("struct FunT {")
    w("  double T;")
    w("  double cvk[%d], u[%d];" % (kk, kk))
    w("  double k[%d];   // forward rate constants, then" % len(arr))
    if rev:
        w("                 // reverse: " + ", ".join("k[%d] of reaction %d" % (kr_at[i], i) for i in rev))
    if fall:
        w("                 // low- over high-pressure: " +
          ", ".join("k[%d] of reaction %d" % (lo_at[i], i) for i in fall))
    if troe:
        w("  double lnfc[%d], trc[%d], trn[%d];   // reactions %s" % ((len(troe),) * 3 + (", ".join(map(str, troe)),)))
    w("};")
    w("")
    w("HD __forceinline__ void cell_set(double rho, Cell<%d>& c) {" % kk)
    w("  c.rho = rho;")
    w("  c.rho_i = c_rcp(rho);")
    for k in range(kk):
        w("  c.rw[%d] = rho * %s;" % (k, lit(wt_inv[k])))
    w("}")
    w("")
    # ---------------------------------------------------------------- tables
    w("// A, b, E/R of the Arrhenius expressions; c_v (5) and internal energy (6)")
    w("// polynomials of the species below and above their middle temperature: in")
    w("// constant memory, so that the loops over them stay small code")
    rows = ["{%s}" % ", ".join(lit(x) for x in p) for p in arr[:n_exp]]
    nasa = []
    for q in range(2):
        sp = []
        for k in range(kk):
            a = list(m.a[k][q])
            c = [ru_wt[k] * (a[0] - 1.0)] + [ru_wt[k] * a[j] for j in range(1, 5)]
            e = [m.ru * (a[0] - 1.0)] + [m.ru * a[j] / float(j + 1) for j in range(1, 5)] + [m.ru * a[5]]
            sp.append("{%s}" % ", ".join(lit(x) for x in c + e))
        nasa.append("{%s}" % ",\\\n   ".join(sp))
    w("#define CHEM_GEN_ARR %s" % ", \\\n  ".join(rows))
    w("#define CHEM_GEN_NASA %s" % ", \\\n  ".join(nasa))
    w("__constant__ double arr_dev[%d][3] = {CHEM_GEN_ARR};" % n_exp)
    w("__constant__ double nasa_dev[2][%d][11] = {CHEM_GEN_NASA};" % kk)
    w("#ifdef __CUDA_ARCH__")
    w("#define CHEM_GEN_TAB(x) x##_dev")
    w("#else")
    w("static const double arr_host[%d][3] = {CHEM_GEN_ARR};" % n_exp)
    w("static const double nasa_host[2][%d][11] = {CHEM_GEN_NASA};" % kk)
    w("#define CHEM_GEN_TAB(x) x##_host")
    w("#endif")
    w("")
    # ---------------------------------------------------------------- tpart
    w("HD __forceinline__ void tpart(double T, FunT& t) {")
    w("  const double Tinv = c_rcp(T);")
    w("  const double alogt = c_log(T);")
    w("  t.T = T;")
    if eqk:
        w("  const double T2 = T * T, T3 = T * T2, T4 = T2 * T2;")
        w("  double %s;   // S/R - H/RT (CKSMH)" % ", ".join("smh%d" % k for k in range(kk)))
    tm = sorted(set(m.tmid[k] for k in range(kk)))
    for q, x in enumerate(tm):
        w("  const int hi%d = T > %s ? 1 : 0;" % (q, lit(x)))
    for k in range(kk):
        lo, hi = list(m.a[k][0]), list(m.a[k][1])
        w("  {   // species %d" % k)
        w("    const double* c = CHEM_GEN_TAB(nasa)[hi%d][%d];" % (tm.index(m.tmid[k]), k))
        w("    t.cvk[%d] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));" % k)
        w("    t.u[%d] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));" % k)
        if eqk:
            for j in range(7):
                w("    const double a%d = hi%d ? %s : %s;" % (j, tm.index(m.tmid[k]), lit(hi[j]), lit(lo[j])))
            w("    const double sv = (alogt - 1.0) * a0 + (0.5 * T) * a1 + (T2 * (1.0 / 6.0)) * a2 +")
            w("                      (T3 * (1.0 / 12.0)) * a3 + (T4 * 0.05) * a4;")
            w("    smh%d = sv + a6 - a5 * Tinv;" % k)
        w("  }")
    w("#pragma unroll 2")
    w("  for (int i = 0; i < %d; ++i) {" % n_exp)
    w("    const double* p = CHEM_GEN_TAB(arr)[i];")
    w("    t.k[i] = p[0] * fm_exp(p[1] * alogt - p[2] * Tinv);")
    w("  }")
    for r in R:
        i = r["i"]
        if any(r["lt"]):   # Landau-Teller: the expression of fun_tpart
            w("  t.k[%d] = t.k[%d] * c_exp(%s / pow(T, %s) + %s / pow(T, %s));"
              % (i, i, lit(r["lt"][0]), lit(LT_P1), lit(r["lt"][1]), lit(LT_P2)))
        if r["rev"] == 1:   # k_f / K_c, K_c from the species' S/R - H/RT
            w("  {")
            w("    double sumsmh = 0.0;")
            for n in range(6):
                if r["nuk"][n] >= 0:
                    w("    sumsmh = sumsmh + %s * smh%d;" % (lit(float(r["nu"][n])), r["nuk"][n]))
            w("    double eqk = sumsmh != 0.0 ? c_exp(fmin(sumsmh, 690.77552789821368)) : 1.0;")
            w("    eqk = eqk * powi(%s * Tinv / %s, %d);" % (lit(m.patm), lit(m.ru), sum(r["nu"])))
            w("    t.k[%d] = c_div(t.k[%d], fmax(eqk, 1.0e-300));" % (kr_at[i], i))
            w("  }")
        if any(r["rlt"]):
            w("  t.k[%d] = t.k[%d] * c_exp(%s / pow(T, %s) + %s / pow(T, %s));"
              % (kr_at[i], kr_at[i], lit(r["rlt"][0]), lit(LT_P1), lit(r["rlt"][1]), lit(LT_P2)))
        if r["fall"]:
            w("  t.k[%d] = c_div(t.k[%d], t.k[%d]);" % (lo_at[i], lo_at[i], i))
            if r["fall"] == 2:   # SRI: ln(a exp(-b/T) + exp(-T/c)) in the lnfc slot
                sr = r["sri"]
                cinv = 1.0 / sr[2] if sr[2] != 0.0 else 0.0
                w("  t.lnfc[%d] = c_log(%s * c_exp(-%s * Tinv) + c_exp(-T * %s));" % (tr_slot[i], lit(sr[0]), lit(sr[1]),
                                                                                  lit(cinv)))
            elif r["fall"] > 1:
                ta = r["troe"][0]
                ti0 = 1.0 / r["troe"][1] if r["troe"][1] != 0.0 else 0.0
                ti1 = 1.0 / r["troe"][2] if r["troe"][2] != 0.0 else 0.0
                w("  {")
                w("    const double ta = %s;" % lit(ta))
                w("    double fcent = (1.0 - ta) * c_exp(-T * %s) + ta * c_exp(-T * %s);" % (lit(ti0), lit(ti1)))
                if r["fall"] == 4:
                    w("    fcent = fcent + c_exp(-%s * Tinv);" % lit(r["troe"][3]))
                w("    const double lnfc = c_log(fmax(fcent, 1.0e-300));")
                w("    t.lnfc[%d] = lnfc;" % tr_slot[i])
                w("    t.trc[%d] = kTroeC + 0.67 * lnfc;" % tr_slot[i])
                w("    t.trn[%d] = kTroeN - 1.27 * lnfc;" % tr_slot[i])
                w("  }")
    w("}")
    w("")
    # ---------------------------------------------------------------- cpart
    w("HD __forceinline__ void cpart(const Cell<%d>& cell, const double* z, const FunT& t, double* zp) {" % kk)
    w("  const double* Y = z + 1;")
    w("  double cv = 0.0, ctot = 0.0;")
    for k in range(kk):
        w("  cv = cv + Y[%d] * t.cvk[%d];" % (k, k))
        w("  const double C%d = Y[%d] * cell.rw[%d];" % (k, k, k))
        w("  ctot = ctot + C%d;" % k)
    for r in R:
        i = r["i"]
        nuk, nu = r["nuk"], r["nu"]
        w("  double rop%d;" % i)
        w("  {   // reaction %d" % i)
        w("    double rkft = t.k[%d];" % i)
        isrev = r["rev"] != 0
        if isrev:
            w("    double rkrt = t.k[%d];" % kr_at[i])
        ctb = None
        if r["thb"]:
            w("    double ctb = ctot;")
            for k in range(kk):
                if r["eff"][k] != 1.0:
                    w("    ctb = ctb + %s * C%d;" % (lit(r["eff"][k] - 1.0), k))
            ctb = "ctb"
        if r["fall"]:
            if r["kfal"]:   # one species is the collider; a third-body factor stays
                w("    const double pr = t.k[%d] * C%d;" % (lo_at[i], r["kfal"] - 1))
            else:
                w("    const double pr = t.k[%d] * %s;" % (lo_at[i], ctb if ctb else "1.0"))
                ctb = None
            w("    double pcor = c_div(pr, 1.0 + pr);")
            if r["fall"] == 2:
                w("    {")
                w("      const double prlog = c_log(fmax(pr, 1.0e-300)) * kInvLn10;")
                w("      const double xp = c_rcp(1.0 + prlog * prlog);")
                w("      pcor = c_exp(xp * t.lnfc[%d]) * %s * pow(t.T, %s) * pcor;" % (tr_slot[i], lit(r["sri"][3]),
                                                                                   lit(r["sri"][4])))
                w("    }")
            elif r["fall"] > 1:
                w("    pcor = troe_factor(pr, t.lnfc[%d], t.trc[%d], t.trn[%d]) * pcor;" % ((tr_slot[i],) * 3))
            w("    rkft = rkft * pcor;")
            if isrev:
                w("    rkrt = rkrt * pcor;")
        if ctb:
            w("    rkft = rkft * ctb;")
            if isrev:
                w("    rkrt = rkrt * ctb;")
        w("    double rkf = rkft * %s;" % powi_expr("C%d" % nuk[0], -nu[0]))
        if isrev:
            w("    double rkr = rkrt * %s;" % powi_expr("C%d" % nuk[3], nu[3]))
        if nuk[1] >= 0:
            w("    rkf = rkf * %s;" % powi_expr("C%d" % nuk[1], -nu[1]))
            if nuk[2] >= 0:
                w("    rkf = rkf * %s;" % powi_expr("C%d" % nuk[2], -nu[2]))
        if isrev and nuk[4] >= 0:
            w("    rkr = rkr * %s;" % powi_expr("C%d" % nuk[4], nu[4]))
            if nuk[5] >= 0:
                w("    rkr = rkr * %s;" % powi_expr("C%d" % nuk[5], nu[5]))
        w("    rop%d = %s;" % (i, "rkf - rkr" if isrev else "rkf"))
        w("  }")
    # production rates, in the generic accumulation order (slot outer, reaction inner)
    acc = {k: [] for k in range(kk)}
    for n in range(6):
        for r in R:
            k = r["nuk"][n]
            if k >= 0:
                v = r["nu"][n]
                acc[k].append("%s rop%d%s" % ("+" if v > 0 else "-", r["i"],
                                              "" if abs(v) == 1 else " * %s" % lit(float(abs(v)))))
    for k in range(kk):
        expr = " ".join(acc[k]) if acc[k] else "0.0"
        w("  const double wdot%d = %s;" % (k, expr))
    w("  double sum = 0.0;")
    for k in range(kk):
        if not acc[k]:   # an inert species
            w("  zp[%d] = 0.0;" % (k + 1))
            continue
        w("  zp[%d] = wdot%d * %s * cell.rho_i;" % (k + 1, k, lit(m.wt[k])))
        w("  sum = sum + t.u[%d] * wdot%d;" % (k, k))
    w("  zp[0] = -c_div(sum, cell.rho * cv);")
    w("}")
    w("")
    w("// the same from the density alone")
    w("HD __forceinline__ void cpart(double rho, const double* z, const FunT& t, double* zp) {")
    w("  Cell<%d> cell;" % kk)
    w("  cell_set(rho, cell);")
    w("  cpart(cell, z, t, zp);")
    w("}")
    w("")
    # ------------------------------------------------------- host check
    w("// True when m is the mechanism this file was generated from (every table")
    w("// entry the right-hand side reads, bit for bit).")
    w("inline bool matches(const izem_mech& m) {")
    w("  auto b = [](double x) { unsigned long long u; memcpy(&u, &x, sizeof(u)); return u; };")
    w("  if (m.kk != %d || m.ii != %d || b(m.ru) != %s) return false;" % (kk, m.ii, bits(m.ru)))
    conds = []
    for k in range(kk):
        conds.append("b(m.wt[%d]) == %s" % (k, bits(m.wt[k])))
        conds.append("b(m.tmid[%d]) == %s" % (k, bits(m.tmid[k])))
        for s_ in range(2):
            for j in range(7):
                conds.append("b(m.a[%d][%d][%d]) == %s" % (k, s_, j, bits(m.a[k][s_][j])))
    for r in R:
        i = r["i"]
        for n in range(6):
            conds.append("m.nuk[%d][%d] == %d && m.nu[%d][%d] == %d" % (i, n, r["nuk"][n], i, n, r["nu"][n]))
        for j in range(3):
            conds.append("b(m.par[%d][%d]) == %s" % (i, j, bits(r["par"][j])))
        conds.append("m.rev[%d] == %d && m.thb[%d] == %d && m.fall[%d] == %d" % (i, r["rev"], i, r["thb"], i, r["fall"]))
        for j in range(2):
            conds.append("b(m.lt[%d][%d]) == %s && b(m.rlt[%d][%d]) == %s" % (i, j, bits(r["lt"][j]), i, j,
                                                                          bits(r["rlt"][j])))
        if r["rev"] == 2:
            for j in range(3):
                conds.append("b(m.rpar[%d][%d]) == %s" % (i, j, bits(r["rpar"][j])))
        if r["thb"]:
            for k in range(kk):
                conds.append("b(m.eff[%d][%d]) == %s" % (i, k, bits(r["eff"][k])))
        if r["fall"]:
            conds.append("m.kfal[%d] == %d" % (i, r["kfal"]))
            for j in range(3):
                conds.append("b(m.low[%d][%d]) == %s" % (i, j, bits(r["low"][j])))
            if r["fall"] == 2:
                for j in range(5):
                    conds.append("b(m.sri[%d][%d]) == %s" % (i, j, bits(r["sri"][j])))
            elif r["fall"] > 1:
                for j in range(4 if r["fall"] == 4 else 3):
                    conds.append("b(m.troe[%d][%d]) == %s" % (i, j, bits(r["troe"][j])))
    for q in range(0, len(conds), 4):
        w("  if (!(%s)) return false;" % " && ".join(conds[q:q + 4]))
    w("  return true;")
    w("}")
    w("")
    w("}  // namespace chem_gen")
    return "\n".join(L) + "\n"


def main():
    from .mech import h2_mechanism
    text = generate(h2_mechanism())
    with open(OUT, "w") as f:
        f.write(text)
    print("wrote %s (%d lines)" % (OUT, text.count("\n")))


if __name__ == "__main__":
    main()
