"""Regenerate ``wvl_composed.h``, the taps of the composed operators that the
fused kernels use (wvlh_lines.cuh), B = magic filter . synthesis and T = analysis .
kinetic . synthesis, from the filters of ``wvl_filters.h``.

B.  The exact taps gs(m), gw(m), m in [-14, 16], are sums of products of the
filters' doubles, taken here as rationals.  Storing a tap moves it by up to half
a rounding, the same way for every output, and so moves |B x|^2, and with it
E_pot and the density, by <x | (B^T D + D^T B) x>, D the taps' errors, whatever
the orbital.  Only 31 of the 62 directions of D do that (to first order the
others turn B x and leave its length).  So the taps are rounded one after the
other, the largest first, each to the neighbour of what the least-squares
solution for the taps still free asks of it: the least norm of
B^T D + D^T B over all frequencies, plus LAMBDA |D|^2, which keeps D small.

FP32 taps are kept times NORM, whose -6th power the kernels multiply back (the
potential's term, E_pot and the density hold six B each): found by a scan of
[2^-1/2, 2^1/2] in steps of 1e-10 among the factors whose taps lie nearest to
FP32 values and whose -6th power lies within 2e-9 of one.  Its four largest taps
take their nearest values, and a local search over the next thirty (steps of a
few roundings, seeded) balances what measure() returns.

T.  Its taps a(l), c(l), e(l), l in [-14, 14], are taken from the same doubles
(the operator that the filters of the separate passes amount to; the published
tables of a, c, e are that of the filters' many-digit values, whose scaling part
differs by 1e-15 at zero frequency, where a smooth orbital's kinetic energy has
nothing else).  Their errors D enter E_kin as <x | D x>, so they are
rounded in turn likewise, the norm of D weighted by 1 / (theta^2 + 0.03) in its
scaling-scaling part, where orbitals live.  The taps left out (T_REACH) count
as errors.  FP32 taps are kept times T_NORM, found by a scan like NORM.

Run ``python gen_composed.py`` to rewrite the header; it is committed, so that the
build needs neither this script nor numpy.
"""
import random
import re
from fractions import Fraction
from pathlib import Path

import numpy as np

HERE = Path(__file__).resolve().parent
NORM = {64: 1.0, 32: 0.9752083272817533}
BITS = {64: 53, 32: 24}
LAMBDA = {64: 0.01, 32: 0.1}
KEEP = {64: 0, 32: 4}
TH = np.linspace(0.0, np.pi, 129)


def table(name):
    t = re.search(r"#define WVL_%s_INIT \{(.*?)\}" % name, (HERE / "wvl_filters.h").read_text(), re.S).group(1)
    return [Fraction(float(v)) for v in t.replace("\\", "").split(",")]


def exact_taps():
    """[gs(-14..16) | gw(-14..16)] as rationals"""
    mf = table("MF")
    return [sum((mf[l + 8] * f[m + l + 7] for l in range(-8, 8) if 0 <= m + l + 7 <= 15), Fraction(0))
            for f in (table("CH"), table("CG")) for m in range(-14, 17)]


def symbols():
    """E[i]: the 2 x 2 symbol (output parity, input half) of tap i on TH"""
    E = np.zeros((62, len(TH), 2, 2), complex)
    for i in range(62):
        half, m = i // 31, i % 31 - 14
        E[i, :, m & 1, half] = np.exp(-1j * TH * ((m - (m & 1)) // 2))
    return E


E = symbols()
EXACT = exact_taps()
HERM = np.einsum("toa,itob->itab", np.tensordot(np.array([float(c) for c in EXACT]), E, 1).conj(), E)
HERM = HERM + np.conj(np.swapaxes(HERM, 2, 3))     # tap i's share of B^T D + D^T B


def rounded(x, bits):
    """the rational x to `bits` binary digits"""
    q = Fraction(2) ** (int(np.floor(np.log2(abs(float(x))))) + 1 - bits)
    return round(x / q) * q


def error(tap, i, prec):
    return float(tap / Fraction(NORM[prec]) - EXACT[i])


def measure(d):
    """of B^T D + D^T B: the largest eigenvalue, the largest and the
    zero-frequency scaling-scaling entry (smooth lines), the mean (white noise);
    and the largest |D|"""
    M, D = np.tensordot(d, HERM, 1), np.tensordot(d, E, 1)
    a, b = M[:, 0, 0].real, M[:, 1, 1].real
    return np.array([np.abs(np.linalg.eigvalsh(M)).max(), np.abs(a[TH < 1]).max(), abs(a[0]), abs((a + b).mean() / 2),
                     np.linalg.norm(D, 2, axis=(1, 2)).max()])


ORDER = sorted(range(62), key=lambda i: -abs(EXACT[i]))


def in_turn(A, exact, order, prec, norm, lam, keep, taps, d):
    """Round the taps of `order` one after the other (the first `keep` to the
    nearest value), A d = the errors' weighted symbols; taps and their errors d
    are filled in"""
    A = np.vstack([A, np.sqrt(lam) * np.eye(len(exact))])
    for k, i in enumerate(order):
        want = 0.0 if k < keep else np.linalg.lstsq(A[:, order[k:]], -A @ d, rcond=None)[0][0]
        taps[i] = rounded(Fraction(norm) * (exact[i] + Fraction(want)), BITS[prec])
        d[i] = float(taps[i] / Fraction(norm) - exact[i])
    return taps


def b_taps(prec):
    A = np.stack([HERM[:, :, 0, 0].real, HERM[:, :, 1, 1].real, np.sqrt(2) * HERM[:, :, 0, 1].real,
                  np.sqrt(2) * HERM[:, :, 0, 1].imag], 2).reshape(62, -1).T / np.sqrt(len(TH))
    taps = in_turn(A, EXACT, ORDER, prec, NORM[prec], LAMBDA[prec], KEEP[prec], [None] * 62, np.zeros(62))
    return refine(taps, prec) if prec == 32 else taps


def refine(taps, prec):
    goal = np.array([2.4e-9, 1.2e-9, 6e-10, 3e-10, 8e-9])
    cost = lambda t: ((measure(np.array([error(v, i, prec) for i, v in enumerate(t)])) / goal) ** 4).sum()  # noqa: E731
    rng, best, idle = random.Random(1), cost(taps), 0
    while idle < 3000:
        t = list(taps)
        for i in rng.sample(ORDER[4:34], rng.choice((1, 1, 2, 2, 3))):
            ulp = Fraction(2) ** (int(np.floor(np.log2(abs(float(t[i]))))) + 1 - BITS[prec])
            t[i] += rng.choice((-1, 1)) * (1 if ulp > 2e-9 else rng.choice((1, 1, 2, 4, 8))) * ulp
        c = cost(t)
        taps, best, idle = (t, c, 0) if c < best else (taps, best, idle + 1)
    return taps


T_NORM = {64: 1.0, 32: 1.9474363232066856}
T_REACH = {64: 13, 32: 11}
T_TAPS = [("A", l) for l in range(15)] + [("C", l) for l in range(-14, 15)] + [("E", l) for l in range(15)]


def t_exact():
    """a(0..14), c(-14..14), e(0..14) of 4 analysis . kinetic . synthesis (the
    kinetic filter is that of the fine spacing)"""
    kin, fine = table("KIN"), (table("CH"), table("CG"))
    line = []          # kinetic . synthesis of a unit scaling / wavelet coefficient
    for f in fine:
        y = [Fraction(0)] * 60
        for p in range(16):
            for l in range(-14, 15):
                y[p + l + 22] += kin[abs(l)] * f[p]
        line.append(y)
    # output half o at coarse distance l from the input (half i): 2 l + p
    at = lambda o, i, l: 4 * sum((fine[o][p] * line[i][2 * l + p + 22] for p in range(16)  # noqa: E731
                                  if 0 <= 2 * l + p + 22 < 60), Fraction(0))
    return [at(*{"A": (0, 0, l), "E": (1, 1, l), "C": (1, 0, -l)}[k]) for k, l in T_TAPS]


def t_taps(prec):
    exact, n = t_exact(), len(T_TAPS)
    S = np.zeros((n, 4, len(TH)))      # scaling-scaling, scaling-wavelet (complex), wavelet-wavelet symbols
    for j, (k, l) in enumerate(T_TAPS):
        if k == "C":
            S[j, 1], S[j, 2] = np.cos(TH * l), np.sin(TH * l)
        else:
            S[j, 0 if k == "A" else 3] = (1 if l == 0 else 2) * np.cos(TH * l)
    w = 1 / (TH ** 2 + 0.03)
    A = (S * np.array([w / np.sqrt((w * w).mean()), 0 * w + 1, 0 * w + 1, 0 * w + 1])).reshape(n, -1).T / np.sqrt(len(TH))
    out = [abs(l) > T_REACH[prec] for _, l in T_TAPS]
    taps = [Fraction(0)] * n
    d = np.array([float(-c) if o else 0.0 for c, o in zip(exact, out)])
    order = sorted((j for j in range(n) if not out[j]), key=lambda j: -abs(exact[j]))
    in_turn(A, exact, order, prec, T_NORM[prec], 1e-3, 0, taps, d)
    D = np.tensordot(d, S, 1)
    print("T FP%d scaling part at theta = 0 %.1e, below 0.5 %.1e, below 1 %.1e" %
          (prec, abs(D[0, 0]), np.abs(D[0, TH < 0.5]).max(), np.abs(D[0, TH < 1]).max()))
    return taps


def define(name, comment, taps, prec):
    return ["/* %s */" % comment, "#define WVL_%s_INIT { \\" % name,
            ", \\\n".join("    %s%s" % (float(t).hex(), "f" * (prec == 32)) for t in taps) + "}"]


def render():
    out = ["/* Generated by gen_composed.py from wvl_filters.h; do not edit. */", "#pragma once", ""]
    times = lambda v: ", times %r" % v if v != 1 else ""  # noqa: E731
    for prec in (64, 32):
        taps = b_taps(prec)
        print("B FP%d" % prec, *("%.1e" % v for v in measure(np.array([error(t, i, prec) for i, t in enumerate(taps)]))))
        for k, half in enumerate("SW"):
            out += define("B%d_%s" % (prec, half), "FP%d taps g%s(-14..16) of magic filter . synthesis%s (index m+14)"
                          % (prec, half.lower(), times(NORM[prec])), taps[31 * k:31 * k + 31], prec)
    out += ["/* that factor's -6th power */", "#define WVL_B32_INV6 %s" % float(Fraction(NORM[32]) ** -6).hex()]
    for prec in (64, 32):
        taps = t_taps(prec)
        for k, what in (("A", "a(0..14)"), ("C", "c(-14..14)"), ("E", "e(0..14)")):
            out += define("T%d_%s" % (prec, k), "FP%d taps %s of analysis . kinetic . synthesis%s%s"
                          % (prec, what, times(T_NORM[prec]), " (index l+14)" if k == "C" else ""),
                          [t for t, (q, _) in zip(taps, T_TAPS) if q == k], prec)
    out += ["/* that factor */", "#define WVL_T32_NORM %r" % T_NORM[32]]
    return "\n".join(out) + "\n"


if __name__ == "__main__":
    (HERE / "wvl_composed.h").write_text(render())
