"""Generate log2_lane_table.inc: the 32-entry reduction table of log2_lane in fullrank_fast.cuh, one
entry per lane of a warp.

Entry j serves mantissas m within 1/64 of the centre 1 + j/32: inv_j is 1/(1 + j/32) rounded to 21
significant bits (a double whose low word is zero, so that one 32-bit word holds it and the product
with a 24-bit mantissa is exact), tab_j = -log2(inv_j) evaluated with 60 significant digits and
rounded once to double.  log2(m) = tab_j + log2(m*inv_j) holds exactly for the stored inv_j; entry 0 is
(1, 0), which keeps the logarithm relatively accurate around 1.

    python adafactor-8bit_b200/csrc/gen_log2_lane_table.py > adafactor-8bit_b200/csrc/log2_lane_table.inc
"""
from decimal import Decimal, getcontext
from fractions import Fraction
from struct import pack

getcontext().prec = 60
LN2 = Decimal(2).ln()


def main():
    print("// generated by gen_log2_lane_table.py: { high word of inv_j, tab_j }")
    for j in range(32):
        inv = Fraction(round(Fraction(32, 32 + j) * 2 ** 21), 2 ** 21)
        tab = -((Decimal(inv.numerator) / Decimal(inv.denominator)).ln() / LN2)
        bits = int.from_bytes(pack(">d", float(inv)), "big")
        assert bits & 0xffffffff == 0
        print(f"    {{ 0x{bits >> 32:08x}u, {(abs(float(tab))).hex()} }},")


if __name__ == "__main__":
    main()
