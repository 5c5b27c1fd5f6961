"""Constants of the opacity kernels' table-driven exp (slg_device.cuh).

    python superlite_b200/csrc/exp_table.py

Prints, from 60-digit decimal arithmetic, each the double nearest the exact
value: N/ln2 and what that leaves of it; the Taylor coefficients (ln2/N)^k / k!
of 2^(f/N), k = 1..5; and 2^(j/N), j = 0..N-1.  The header's constants are
this output for N = 64.
"""
import math
from decimal import Decimal, getcontext

N = 64


def constants():
    getcontext().prec = 60
    q = Decimal(2).ln() / N
    inv = 1 / q
    return {"inv_l": float(inv), "inv_lo": float(inv - Decimal(float(inv))),
            "taylor": [float(q ** k / math.factorial(k)) for k in range(1, 6)],
            "table": [float(Decimal(2) ** (Decimal(j) / N)) for j in range(N)]}


def main():
    c = constants()
    print(f"kExpInvL = {c['inv_l']!r}  kExpInvLLo = {c['inv_lo']!r}")
    print(f"c1..c5 = {c['taylor']}")
    t = c["table"]
    for k in range(0, N, 4):
        print("    " + ", ".join(repr(v) for v in t[k:k + 4]) + ",")


if __name__ == "__main__":
    main()
