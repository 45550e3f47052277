"""Writes w<L>.inc: exp(-2 pi i m / L), m = 0..L-1, as 21-digit decimal literals.

96 is divisible by the in-register DFT sizes 2, 3, 4, 8, 12, 16, 24 and 32 of the
line FFTs, 160 by 5, 20 and 40: wk<K>(m) = W_L^(m * L / K).  The values are
computed with Python's decimal module at 40 digits (pi from Machin's formula,
cos and sin from their Taylor series), so every literal is correctly rounded.

    python gen_w96.py > w96.inc
    python gen_w96.py 160 > w160.inc
"""
import sys
from decimal import Decimal, getcontext

getcontext().prec = 40


def arctan_inv(x):
    """arctan(1/x) for integer x by its Taylor series."""
    x = Decimal(x)
    x2 = x * x
    term = Decimal(1) / x
    total, n, sign = term, 1, 1
    while True:
        term /= x2
        n += 2
        sign = -sign
        t = term / n
        if t < Decimal(10) ** -45:
            return total
        total += sign * t


PI = 4 * (4 * arctan_inv(5) - arctan_inv(239))


def cos_sin(a):
    c, s = Decimal(0), Decimal(0)
    term, k = Decimal(1), 0
    while abs(term) > Decimal(10) ** -45:
        if k % 4 == 0:
            c += term
        elif k % 4 == 1:
            s += term
        elif k % 4 == 2:
            c -= term
        else:
            s -= term
        k += 1
        term = term * a / k
    return c, s


def lit(v):
    if v == 0:
        return "0.0"
    q = f"{v:.21f}".rstrip("0")
    return q + "0" if q.endswith(".") else q


def main():
    L = int(sys.argv[1]) if len(sys.argv) > 1 else 96
    re, im = [], []
    for m in range(L):
        c, s = cos_sin(2 * PI * m / L)
        if m % (L // 4) == 0:
            c, s = [Decimal(1), Decimal(0), Decimal(-1), Decimal(0)][m // (L // 4)], [Decimal(0), Decimal(1), Decimal(0), Decimal(-1)][m // (L // 4)]
        re.append(c)
        im.append(-s)
    out = [f"// exp(-2*pi*i*m/{L}) = w{L}re(m) + i*w{L}im(m); exact decimal literals (21 digits), from gen_w96.py."]
    for name, vals in ((f"w{L}re", re), (f"w{L}im", im)):
        out.append(f"DDB_HD constexpr double {name}(int m) {{")
        out.append(f"  switch (((m % {L}) + {L}) % {L}) {{")
        for m, v in enumerate(vals):
            out.append(f"    case {m}: return {lit(v)};")
        out.append("    default: return 0.0;")
        out.append("  }")
        out.append("}")
    print("\n".join(out))


if __name__ == "__main__":
    main()
