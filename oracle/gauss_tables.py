"""The constants of the FP64 Box-Muller transform (csrc/gauss64.cuh), from their definitions in
50-digit decimal arithmetic:

* ``log_table(n)``: n intervals of [0.6875, 1.375) that split the high words of its doubles evenly;
  per interval the reciprocal c of its centre rounded to a high word (1 for the last interval
  below 1) and T = 2 ln c, its part above 2^-40 and the high word of the rest (P. T. P. Tang, ACM
  TOMS 16, 1990);
* ``log_step()``: -2 ln 2 as a multiple of 2^-40 and the double nearest to the rest;
* ``sine()``: P of sin y = y + y^3 P(y^2), interpolated at the eight Chebyshev nodes of y^2 in
  [0, (pi/2)^2], from the highest coefficient down.

``python -m oracle.gauss_tables [n]`` prints the table as it stands in the source."""
import decimal as D
import struct
import sys

D.getcontext().prec = 60
PI = D.Decimal("3.14159265358979323846264338327950288419716939937510582097494459")


def bits(x: float) -> int:
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def from_bits(b: int) -> float:
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def high_word(x) -> int:
    """The double nearest to x, rounded to the nearest high word."""
    return (bits(float(x)) + (1 << 31)) >> 32


def split40(x):
    """(the multiple of 2^-40 nearest to x, the rest)"""
    head = (x * 2 ** 40).to_integral_value(D.ROUND_HALF_EVEN) / 2 ** 40
    return head, x - head


def log_table(n=128):
    step = (1 << 20) // n
    rows = []
    for q in range(n):
        lo = (0x3FE60000 + q * step) << 32
        a, b = D.Decimal(from_bits(lo)), D.Decimal(from_bits(lo + (step << 32)))
        c = 0x3FF00000 if b == 1 else high_word(2 / (a + b))
        head, rest = split40(2 * D.Decimal(from_bits(c << 32)).ln())
        rows.append((bits(float(head)), high_word(rest) << 32 | c))
    return rows


def log_step():
    head, rest = split40(-2 * D.Decimal(2).ln())
    return float(head), float(rest)


def _sin(y):
    term = total = y
    k = 1
    while abs(term) > D.Decimal(10) ** -58:
        term = -term * y * y / ((k + 1) * (k + 2))
        total += term
        k += 2
    return total


def _cos(y):
    term = total = D.Decimal(1)
    k = 0
    while abs(term) > D.Decimal(10) ** -58:
        term = -term * y * y / ((k + 1) * (k + 2))
        total += term
        k += 2
    return total


def sine(n=8):
    top = (PI / 2) ** 2
    t = [top / 2 * (1 + _cos((2 * q + 1) * PI / (2 * n))) for q in range(n)]
    div = [(_sin(x.sqrt()) - x.sqrt()) / (x * x.sqrt()) for x in t]
    for k in range(1, n):                      # Newton's divided differences
        for q in range(n - 1, k - 1, -1):
            div[q] = (div[q] - div[q - 1]) / (t[q] - t[q - k])
    poly = [D.Decimal(0)] * n                  # ascending powers
    for q in range(n - 1, -1, -1):
        poly = [(poly[k - 1] if k else 0) - t[q] * poly[k] for k in range(n)]
        poly[0] += div[q]
    return [float(c) for c in reversed(poly)]


if __name__ == "__main__":
    out = ["{0x%016x, 0x%016x}" % r for r in log_table(int(sys.argv[1]) if len(sys.argv) > 1 else 128)]
    for q in range(0, len(out), 2):
        print("    " + ", ".join(out[q:q + 2]) + ",")
    print("//", *[x.hex() for x in log_step()])
    print("//", *[x.hex() for x in sine()])
