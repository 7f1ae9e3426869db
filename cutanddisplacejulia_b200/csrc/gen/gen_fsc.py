"""Generate ../fsc_rows.cuh: the free-surface correction of a triangle side as
fixed linear combinations of few harmonic functions.

The correction of an angular dislocation below a free surface (Comninou and
Dundurs 1975; src/TD.jl:1423-1489 for the displacements) is, in the image
coordinates (y1, y2, q), r the image distance, depth z of the point, depth a of
the side's end, inclination beta of the side (s, c its sine and cosine):

    u = sum of  F, log p, log w, powers of zeta and eta          (level 0)
      + (a or z) x  zeta^m / r, eta^m / r                        (level 1)
      + a z x  their derivatives along the axis                  (level 2)

with p = r + q, zeta = (y1 + i y2) / p for the vertical leg and, in the frame
(z1, y2, z3) turned by beta, w = r + z3, eta = (z1 + i y2) / w for the inclined
one.  Table U below holds those coefficients.  The families are closed under
differentiation: with G_0 = log p, G_m = -zeta^m / m, h_m = zeta^m / r and
D = d/dq,  D G_m = h_m,  (d1 + i d2) G_m = h_(m+1),  (d1 - i d2) G_m =
-h_(m-1); so the strain is a linear combination of h_m, D h_m, D^2 h_m too
(tables of at most ten terms instead of several hundred operations per entry),
with the same coefficients at both ends of the side.

The generator differentiates U, reduces the coefficients with c^2 + s^2 = 1,
combines the powers of zeta and eta that always occur together (M, S, Y, O, N
below) and prints the rows and the per-side set-up of their coefficients.
Needs sympy (development time only):  python gen_fsc.py
"""
import os

import sympy as sp

HERE = os.path.dirname(os.path.abspath(__file__))
s, c, nu = sp.symbols("s c nu")
t = c / s
N1, N2, half = 1 - 2 * nu, 2 * (1 - nu), sp.Rational(1, 2)
S = sp.Symbol

# Displacement component i of slip component g: level-0 names, then ('A', .),
# ('Z', .) level-1 functions weighted by a or z, ('AZ', .) level-2 ones; Z / E
# are zeta / eta, h / g their level-1 functions, y1, y2, q over r^3.
U = {
    (1, 1): {"F": -N2 * N1 * t**2, "ImZ1": N1**2 * t, "ImZ2": -N1 * nu / 2, "ImE1": N1 * c**2 * t,
             ("A", "Im_h1"): -N1 * t, ("A", "Im_g1"): N1 * c * t, ("A", "Im_h2"): -N1 / 2, ("Z", "Im_h1"): -N1 * t,
             ("Z", "Im_g1"): c**2 * (N1 * c * t + N2 * s), ("Z", "Im_h2"): nu, ("Z", "Im_g2"): -c**3 / 2,
             ("AZ", "y2"): c * s, ("AZ", "Im_h2"): -half, ("AZ", "Im_g2"): c**2 / 2},
    (1, 2): {"phi": N1 * (N2 * t**2 + nu), "chi": -N1 * (N2 * t**2 + 1) * c, "ReZ1": -N1**2 * t, "ReZ2": N1 * nu / 2,
             "ReE1": -N1 * c * t, ("A", "/r"): N1 / 2, ("A", "Re_h1"): N1 * t, ("A", "Re_g1"): -N1 * t,
             ("A", "Re_h2"): N1 / 2, ("Z", "/r"): nu + (1 - 4 * nu) * c**2 / 2, ("Z", "Re_h1"): N1 * t,
             ("Z", "Re_g1"): -t * (s**2 + N1 * c**2), ("Z", "Re_h2"): -nu, ("Z", "Re_g2"): c**2 / 2,
             ("AZ", "y1"): -c * s / 2, ("AZ", "q"): -s**2 / 2, ("AZ", "Re_h2"): half, ("AZ", "Re_g2"): -c / 2},
    (1, 3): {"ImZ1": N1, "ImE1": -N1 * c**2, ("A", "Im_h1"): N1, ("A", "Im_g1"): -N1 * c, ("Z", "Im_h1"): -1,
             ("Z", "Im_g1"): c**3, ("Z", "Im_g2"): c**2 * s / 2, ("AZ", "y2"): -s**2, ("AZ", "Im_g2"): -c * s / 2},
    (2, 1): {"phi": N1 * (N2 * t**2 - nu), "chi": -N1 * (N2 * t**2 + N1) * c, "ReZ1": -N1**2 * t, "ReZ2": N1 * nu / 2,
             "ReE1": -N1 * c * t, ("A", "/r"): N1 / 2, ("A", "Re_h1"): N1 * t, ("A", "Re_g1"): -N1 * t,
             ("A", "Re_h2"): N1 / 2, ("Z", "/r"): -nu + c**2 / 2, ("Z", "Re_h1"): N1 * t, ("Z", "Re_g1"): -N1 * t,
             ("Z", "Re_h2"): -nu, ("Z", "Re_g2"): c**2 / 2, ("AZ", "y1"): -c * s / 2, ("AZ", "q"): -s**2 / 2,
             ("AZ", "Re_h2"): half, ("AZ", "Re_g2"): -c / 2},
    (2, 2): {"F": N2 * N1 * t**2, "ImZ1": -N1**2 * t, "ImZ2": N1 * nu / 2, "ImE1": -N1 * t, ("A", "Im_h1"): N1 * t,
             ("A", "Im_g1"): -N1 / s, ("A", "Im_h2"): N1 / 2, ("Z", "Im_h1"): N1 * t, ("Z", "Im_g1"): -N1 * c * t,
             ("Z", "Im_h2"): -nu, ("Z", "Im_g2"): c / 2, ("AZ", "Im_h2"): half, ("AZ", "Im_g2"): -half},
    (2, 3): {"chi": -N1 * s, "ReZ1": -N1, "ReE1": N1 * c, ("A", "Re_h1"): -N1, ("A", "Re_g1"): N1,
             ("Z", "/r"): -c * s / 2, ("Z", "Re_h1"): 1, ("Z", "Re_g1"): -1, ("Z", "Re_g2"): -c * s / 2,
             ("AZ", "y1"): s**2 / 2, ("AZ", "q"): -c * s / 2, ("AZ", "Re_g2"): s / 2},
    (3, 1): {"F": N2 * N1 * t, "ImZ1": 2 * N2 * nu, "ImE1": -N2 * c**2, ("A", "Im_h1"): N2, ("A", "Im_g1"): -N2 * c,
             ("Z", "Im_h1"): 2 * nu, ("Z", "Im_g1"): c * (N1 - c**2), ("Z", "Im_g2"): -c**2 * s / 2,
             ("AZ", "y2"): s**2, ("AZ", "Im_g2"): c * s / 2},
    (3, 2): {"phi": -N2 * N1 * t, "chi": N2 * N1 * t * c, "ReZ1": -2 * N2 * nu, "ReE1": N2 * c, ("A", "Re_h1"): -N2,
             ("A", "Re_g1"): N2, ("Z", "/r"): (1 - 4 * nu) * c * s / 2, ("Z", "Re_h1"): -2 * nu,
             ("Z", "Re_g1"): 2 * nu * c**2, ("Z", "Re_g2"): c * s / 2, ("AZ", "y1"): -s**2 / 2, ("AZ", "q"): c * s / 2,
             ("AZ", "Re_g2"): -s / 2},
    (3, 3): {"F": N2, "ImE1": N2 * s * c, ("A", "Im_g1"): N2 * s, ("Z", "Im_g1"): s * (1 + c**2),
             ("Z", "Im_g2"): c * s**2 / 2, ("AZ", "y2"): c * s, ("AZ", "Im_g2"): -s**2 / 2},
}

# ------------------------------------------------- derivatives of the families
h0 = S("h0")
H = {0: (h0, sp.Integer(0)), 1: (S("h1r"), S("h1i")), 2: (S("h2r"), S("h2i")), 3: (S("h3r"), S("h3i"))}
GG = {0: (h0, sp.Integer(0)), 1: (S("g1r"), S("g1i")), 2: (S("g2r"), S("g2i"))}


def level2(X):
    t1, t2, tq = S(X + "t1"), S(X + "t2"), S(X + "tq")
    Dh = {0: (-tq, 0), 1: (-t1, -t2), 2: (S(X + "p2r"), S(X + "p2i")), 3: (S(X + "p3r"), S(X + "p3i"))}
    z1, z3 = c * t1 + s * tq, -s * t1 + c * tq
    Dg = {0: (-z3, 0), 1: (-z1, -t2), 2: (S(X + "w2r"), S(X + "w2i")), 3: (S(X + "w3r"), S(X + "w3i"))}
    return (t1, t2, tq), Dh, Dg


s11, s12, s1q, s22, s2q = [S("s" + k) for k in ("11", "12", "1q", "22", "2q")]   # second derivatives of 1 / r
sqq = -(s11 + s22)
D2h = {0: (sqq, 0), 1: (s1q, s2q), 2: (s11 - s22, 2 * s12), 3: (S("P3r"), S("P3i"))}
_a11 = c * c * s11 + 2 * c * s * s1q + s * s * sqq
_a13 = -s * c * s11 + (c * c - s * s) * s1q + s * c * sqq
D2g = {0: (s * s * s11 - 2 * s * c * s1q + c * c * sqq, 0), 1: (_a13, -s * s12 + c * s2q),
       2: (_a11 - s22, 2 * (c * s12 + s * s2q)), 3: (S("W3r"), S("W3i"))}


def d_family(fam, k, part):
    up, mid = fam[k + 1], fam[k]
    lo = (-fam[k - 1][0], -fam[k - 1][1]) if k >= 1 else (fam[1][0], -fam[1][1])
    d1 = ((up[0] + lo[0]) / 2, (up[1] + lo[1]) / 2)
    dd = (up[0] - lo[0], up[1] - lo[1])
    i = 0 if part == "Re" else 1
    return [d1[i], (dd[1] / 2, -dd[0] / 2)[i], mid[i]]


def from_turned(v):
    return [c * v[0] - s * v[2], v[1], s * v[0] + c * v[2]]


def grad(n):
    """Gradient of a term of U, and what the factor z adds to its q derivative."""
    if isinstance(n, str):
        if n == "F":
            return [H[1][1] - c * GG[1][1], GG[1][0] - H[1][0], -s * GG[1][1]], 0
        if n == "phi":
            return d_family(H, 0, "Re"), 0
        if n == "chi":
            return from_turned(d_family(GG, 0, "Re")), 0
        k = int(n[3])
        v = d_family(H if n[2] == "Z" else GG, k, n[:2])
        v = [-k * x for x in v]
        return (v if n[2] == "Z" else from_turned(v)), 0
    lev, n = n
    if lev == "AZ":
        T, Dh, Dg = level2("A")
        if n in ("y1", "y2", "q"):
            i = ("y1", "y2", "q").index(n)
            return [[-s11, -s12, -s1q], [-s12, -s22, -s2q], [-s1q, -s2q, -sqq]][i], T[i]
        i = 0 if n[:2] == "Re" else 1
        if n[3] == "h":
            return d_family(D2h, 2, n[:2]), Dh[2][i]
        return from_turned(d_family(D2g, 2, n[:2])), Dg[2][i]
    _, Dh, Dg = level2(lev)
    z = 1 if lev == "Z" else 0
    if n == "/r":
        return d_family(Dh, 0, "Re"), z * h0
    k, i = int(n[-1]), 0 if n[:2] == "Re" else 1
    if n[3] == "h":
        return d_family(Dh, k, n[:2]), z * H[k][i]
    return from_turned(d_family(Dg, k, n[:2])), z * GG[k][i]


def reduce(e):
    """Polynomial in s, 1/s, nu and at most the first power of c."""
    e = sp.expand(e)
    out = 0
    for term in sp.Add.make_args(e):
        k = sp.Poly(term * s**8, c).degree() if term.has(c) else 0
        out += sp.expand(term / c**k * (1 - s**2) ** (k // 2) * c ** (k % 2))
    return sp.factor(sp.expand(out))


def strains():
    out = {}
    for g in (1, 2, 3):
        J = []
        for i in (1, 2, 3):
            row = [0, 0, 0]
            for n, co in U[i, g].items():
                G, extra = grad(n)
                for k in range(3):
                    row[k] += co * G[k]
                row[2] += co * extra
            J.append(row)
        for k, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
            out[g - 1, k] = sp.expand((J[i][j] + J[j][i]) / 2)
    return out


def replace_groups(e, g, groups):
    """Replace the terms of each (name, {symbol: weight}) group by its name."""
    out = {}
    for name, parts in groups:
        lead = list(parts)[0]
        co = reduce(e.coeff(S(lead)) / parts[lead])
        if co == 0:
            assert all(reduce(e.coeff(S(x))) == 0 for x in parts), (name, g)
            continue
        for x, w in parts.items():
            assert reduce(e.coeff(S(x)) - co * w) == 0, (name, x, g)
        out[name] = co
        e = sp.expand(e - sum(e.coeff(S(x)) * S(x) for x in parts))
    return e, out


def strain_rows():
    """Per slip and component: {accumulator: coefficient}; names starting with
    'z_' are multiplied by the depth z."""
    rows = {}
    for (g, k), e in strains().items():
        groups = []
        for im in "ri":
            if g < 2:
                groups.append(("M" + im, {"h3" + im: nu * N1 / 2, "Zp3" + im: nu / 2, "Ap3" + im: -N1 / 4, "P3" + im: -sp.Rational(1, 4),
                                          "h2" + im: -t * N1**2 / 2, "Ap2" + im: -t * N1 / 2, "Zp2" + im: -t * N1 / 2}
                               if (k in (0, 1, 3)) else {"Zp2" + im: sp.Integer(1)}))
            else:
                groups.append(("S" + im, {"h2" + im: -N1 / 2, "Ap2" + im: N1 / 2, "Zp2" + im: -half}))
            groups.append(("O" + im, {"Aw2" + im: sp.Integer(1), "g2" + im: -c}))
            groups.append(("N" + im, {"W3" + im: sp.Rational(1, 4), "Zw3" + im: -c / 4}))
        e, row = replace_groups(e, g, groups)
        if g < 2 and k not in (0, 1, 3):   # the lone z D h_2 terms
            row = {("Y" + n[1] if n[0] == "M" else n): (v / nu if n[0] == "M" else v) for n, v in row.items()}
        for x in ("h0", "h1r", "h1i", "g1r", "g1i", "At1", "At2", "Atq"):
            co = reduce(e.coeff(S(x)))
            if co != 0:
                row[x] = co
        for x, n in [("Z" + b, b) for b in ("t1", "t2", "tq", "w2r", "w2i")] + [(b, b) for b in ("s11", "s12", "s1q", "s22", "s2q")]:
            co = reduce(e.coeff(S(x)))
            if co != 0:
                row["z_" + n] = co
            e = sp.expand(e - e.coeff(S(x)) * S(x))
        for x in ("h0", "h1r", "h1i", "g1r", "g1i", "At1", "At2", "Atq"):
            e = sp.expand(e - e.coeff(S(x)) * S(x))
        assert reduce(e) == 0 if e != 0 else True, (g, k, e)
        rows[g, k] = row
    return rows


def disp_rows():
    """d[3 i + g]: component i of slip g.  Accumulators: F, phi, chi; B, B3, B4
    (powers of zeta), O1 = c eta + a g_1, O2 = z (a D g_2 - c g_2), z g_1, a / r,
    z / r and a z (y1, y2, q) / r^3."""
    rows = {}
    for (i, g), u in U.items():
        row = {}
        for n, co in u.items():
            if n in ("F", "phi", "chi"):
                row[n] = co
        im = "i" if any(isinstance(n, str) and n[:2] == "Im" for n in u) else "r"
        R = "Im" if im == "i" else "Re"
        z1 = u.get(R + "Z1")
        if z1 is not None:
            name, w = (("B", N1**2 * t), ("B4", 2 * N2 * nu))[i == 3] if g < 3 else ("B3", N1)
            row[name + im] = z1 / w
        row["O1" + im] = u[("A", R + "_g1")]
        assert sp.simplify(u[R + "E1"] - c * row["O1" + im]) == 0, (i, g)
        row["O2" + im] = u[("AZ", R + "_g2")]
        assert sp.simplify(u[("Z", R + "_g2")] + c * row["O2" + im]) == 0, (i, g)
        row["zg1" + im] = u[("Z", R + "_g1")]
        for n, x in ((("A", "/r"), "ah0"), (("Z", "/r"), "zh0"), (("AZ", "y1"), "azt1"), (("AZ", "y2"), "azt2"),
                     (("AZ", "q"), "aztq")):
            if n in u:
                row[x] = u[n]
        rows[3 * (i - 1) + g - 1] = {k: reduce(v) for k, v in row.items() if reduce(v) != 0}
    return rows


class Coefficients:
    def __init__(self, prefix):
        self.prefix, self.of, self.order = prefix, {}, []

    def term(self, co, name):
        """C text of co * name, with its sign."""
        if co == 1:
            return "+", name
        if co == -1:
            return "-", name
        key = sp.expand(co)
        for sign, k in (("+", key), ("-", sp.expand(-co))):
            if k in self.of:
                return sign, "k.%s * %s" % (self.of[k], name)
        self.of[key] = "%s[%d]" % (self.prefix, len(self.order))
        self.order.append(co)
        return "+", "k.%s * %s" % (self.of[key], name)


def row_text(row, K, pick):
    txt = ""
    for n, co in row.items():
        if not pick(n):
            continue
        sg, body = K.term(co, "a." + n.replace("z_", ""))
        txt += (" %s " % sg if txt else ("-" if sg == "-" else "")) + body
    return txt


def emit():
    K, KD = Coefficients("e"), Coefficients("d")
    srows, drows = strain_rows(), disp_rows()
    body, dbody, nterm = [], [], 0
    for (g, k), row in sorted(srows.items()):
        nterm += len(row)
        p0 = row_text(row, K, lambda n: not n.startswith("z_"))
        p1 = row_text(row, K, lambda n: n.startswith("z_"))
        body.append("    e[%d][%d] = %s%sz * (%s);" % (g, k, p0, " + " if p0 else "", p1))
    for j, row in sorted(drows.items()):
        nterm += len(row)
        dbody.append("    d[%d] = %s;" % (j, row_text(row, KD, lambda n: True)))
    L = ["// GENERATED by csrc/gen/gen_fsc.py -- do not edit.",
         "//", "// Free-surface correction of a triangle side: strain (e[slip][component], tensor",
         "// components 11, 22, 33, 12, 13, 23) and displacement (d[3 component + slip]) in the",
         "// side's coordinates as linear combinations of the accumulators of FscAcc / FscDispAcc",
         "// (end B minus end A), without the factor 1 / (4 pi (1 - nu)).", "#pragma once", "",
         "namespace cad {", ""]
    for name, C in (("FscRows", K), ("FscDispRows", KD)):
        L += ["template <typename T>", "struct %s {" % name]
        L += ["    T %s[%d];" % (C.prefix, len(C.order)), "};", ""]
        L += ["CAD_HD void fsc_rows_setup(double s, double c, double nu, %s<double>& k)" % name, "{",
              "    const double is = 1.0 / s, is2 = is * is;"]
        for co in C.order:
            txt = sp.ccode(sp.factor(co)).replace("(s - 1)*(s + 1)", "(-c*c)")
            for p in (2, 3, 4):
                txt = txt.replace("pow(s, %d)" % p, "(%s)" % "*".join("s" * p))
            txt = txt.replace("/(s*s)", "*is2").replace("/s", "*is")
            txt = txt.replace("(1.0/2.0)", "0.5").replace("1.0/2.0", "0.5").replace("(1.0/4.0)", "0.25").replace(
                "1.0/4.0", "0.25").replace("(3.0/4.0)", "0.75").replace("3.0/4.0", "0.75").replace("5.0/4.0", "1.25")
            L.append("    k.%s = %s;" % (C.of[sp.expand(co)], txt))
        L += ["}", ""]
    L += ["template <typename R>", "CAD_HD void fsc_rows(const FscRows<R>& k, const FscAcc<R>& a, R z, R e[3][6])", "{",
          *body, "}", "", "template <typename R>",
          "CAD_HD void fsc_disp_rows(const FscDispRows<R>& k, const FscDispAcc<R>& a, R d[9])", "{", *dbody, "}", "",
          "}  // namespace cad", ""]
    with open(os.path.join(HERE, "..", "fsc_rows.cuh"), "w") as f:
        f.write("\n".join(L))
    print("terms", nterm, "strain coefficients", len(K.order), "displacement coefficients", len(KD.order))


if __name__ == "__main__":
    emit()
