"""Regenerate ``wvl_composed.h``, the taps of the composed operator B = magic
filter . synthesis that the fused kernels use (wvlh_lines.cuh), from the
filters of ``wvl_filters.h``.

The exact taps gs(m), gw(m), m in [-14, 16], are sums of products of the
filters' doubles, taken here as rationals.  Storing a tap moves it by up to half
a rounding, the same way for every output, and so moves |B x|^2, and with it
E_pot and the density, by <x | (B^T D + D^T B) x>, D the taps' errors, whatever
the orbital.  Only 31 of the 62 directions of D do that (to first order the
others turn B x and leave its length).  So the taps are rounded one after the
other, the largest first, each to the neighbour of what the least-squares
solution for the taps still free asks of it: the least norm of
B^T D + D^T B over all frequencies, plus LAMBDA |D|^2, which keeps D small.

Run ``python gen_composed.py`` to rewrite the header; it is committed, so that the
build needs neither this script nor numpy.
"""
import re
from fractions import Fraction
from pathlib import Path

import numpy as np

HERE = Path(__file__).resolve().parent
LAMBDA = 0.01
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


def least_squares(bits):
    A = np.stack([HERM[:, :, 0, 0].real, HERM[:, :, 1, 1].real, np.sqrt(2) * HERM[:, :, 0, 1].real,
                  np.sqrt(2) * HERM[:, :, 0, 1].imag], 2).reshape(62, -1).T / np.sqrt(len(TH))
    A = np.vstack([A, np.sqrt(LAMBDA) * np.eye(62)])
    free = sorted(range(62), key=lambda i: -abs(EXACT[i]))
    taps, d = [None] * 62, np.zeros(62)
    while free:
        want = np.linalg.lstsq(A[:, free], -A @ d, rcond=None)[0][0]
        i = free.pop(0)
        taps[i] = rounded(EXACT[i] + Fraction(want), bits)
        d[i] = float(taps[i] - EXACT[i])
    return taps


def render():
    out = ["/* Generated by gen_composed.py from wvl_filters.h; do not edit. */", "#pragma once", ""]
    taps = least_squares(53)
    for k, half in enumerate("SW"):
        out += ["/* taps g%s(-14..16) of magic filter . synthesis (index m+14) */" % half.lower(),
                "#define WVL_B64_%s_INIT { \\" % half,
                ", \\\n".join("    %s" % float(t).hex() for t in taps[31 * k:31 * k + 31]) + "}"]
    return "\n".join(out) + "\n"


if __name__ == "__main__":
    (HERE / "wvl_composed.h").write_text(render())
