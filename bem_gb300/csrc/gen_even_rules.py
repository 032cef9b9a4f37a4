"""Writes even_rules.h: weights on the nodes of the 36-point triangle rule
whose moments of degree <= 6 are those of the 91- and 105-point rules as
tabulated (quadrature_tables.h).

The 36-point rule integrates polynomials up to degree 13, but the tables carry
about 12 digits, so its moments differ from the larger rules' by ~1e-12.  The
correction (the least-norm solution of the 28 moment equations, iterated in
exact arithmetic) brings them together to 1e-17 for degrees up to 6 and to
3e-13 up to 13, where the terms that use them are below 1e-7.  Beyond its degree the
rule's moments are off by 1.5e-9 (14) to 5.8e-7 (19); the terms that use those, of the
FP64 series alone, are below 1.1^15/15! = 3e-12.
Run from this directory: python gen_even_rules.py"""
import re
from fractions import Fraction

import numpy as np

TEXT = open("quadrature_tables.h").read()
NUMBER = r"[-+]?(?:\d+\.?\d*|\.\d+)(?:[eE][-+]?\d+)?"


def rule(n):
    body = re.search(r"bemgpu_tri_rule%d\[[^=]*=\s*\{(.*?)\};" % n, TEXT, re.S).group(1)
    vals = [Fraction(float(x)) for x in re.findall(NUMBER, body)]
    return [vals[3 * i:3 * i + 3] for i in range(n)]


nodes = rule(36)
monomials = [(i, d - i) for d in range(7) for i in range(d + 1)]
V = np.array([[float(x) ** i * float(y) ** j for x, y, _ in nodes] for i, j in monomials])
lines = ["// Generated by gen_even_rules.py; do not edit.", "#pragma once", "",
         "// Weights on the nodes of the 36-point rule with the moments (degree <= 6) of",
         "// the 91- and 105-point rules."]
for n in (91, 105):
    target = rule(n)
    w = [q[2] for q in nodes]
    for _ in range(3):
        gap = [float(sum(q[2] * q[0] ** i * q[1] ** j for q in target)
                     - sum(ww * q[0] ** i * q[1] ** j for ww, q in zip(w, nodes))) for i, j in monomials]
        w = [Fraction(float(a + Fraction(float(b)))) for a, b in zip(w, np.linalg.lstsq(V, np.array(gap), rcond=None)[0])]
    lines.append(f"static const double bemgpu_even_w{n}[36] = {{")
    vals = [f"{float(x)!r}" for x in w]
    lines += ["    " + ", ".join(vals[i:i + 4]) + "," for i in range(0, 36, 4)]
    lines.append("};")
open("even_rules.h", "w").write("\n".join(lines) + "\n")
