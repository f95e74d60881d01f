#!/usr/bin/env python3
"""Writes hg_pow_tables.h: the double-double tables of hg_crpow.h.

Every entry is computed here with Python's decimal module at 80 significant
digits and split into a pair (hi, lo) of doubles, hi = the double nearest to
the value, lo = the double nearest to the remainder, so hi + lo carries the
value to about 2^-106 relative:

  LOGC[k + 76] = log(1 + k/256)      k = -76 .. 107   (log argument reduction)
  EXP2[j]      = 2^(j/256)           j = 0 .. 255     (exp argument reduction)
  LN2          = log(2)
  LN2_256      = log(2)/256 as C1 + C2 + C3, C1 with 32 significant bits so
                 that n*C1 is exact for |n| < 2^21
  INV_LN2_256  = 256/log(2) (only selects the reduction index)
  FLOG[i]      = 1/c, -log(1/c) as hi (a multiple of 2^-42) + lo, 0; c the
                 middle of [1 + i/256, 1 + (i+1)/256), but 1 for i = 0 and 2
                 for i = 255; from i = 106 on (c > sqrt 2) less log(2), the
                 exponent being one more there   (quick log)
  FLN2         = log(2) as hi (a multiple of 2^-42) + lo

Usage: python gen_pow_tables.py  (rewrites hg_pow_tables.h beside it)
"""
import os
import struct
from decimal import Decimal, getcontext

getcontext().prec = 80
HERE = os.path.dirname(os.path.abspath(__file__))
K_LO, K_HI = -76, 107


def split(v):
    hi = float(v)
    lo = float(v - Decimal(hi))
    return hi, lo


def truncate_bits(x, bits):
    """x with its significand cut to `bits` significant bits (toward zero)."""
    u = struct.unpack("<Q", struct.pack("<d", x))[0]
    u &= ~((1 << (53 - bits)) - 1)
    return struct.unpack("<d", struct.pack("<Q", u))[0]


def main():
    ln2 = Decimal(2).ln()
    logc = [split((Decimal(1) + Decimal(k) / 256).ln()) for k in range(K_LO, K_HI + 1)]
    exp2 = [split((Decimal(j) / 256 * ln2).exp()) for j in range(256)]
    c = ln2 / 256
    c1 = truncate_bits(float(c), 32)
    c2 = float(c - Decimal(c1))
    c3 = float(c - Decimal(c1) - Decimal(c2))
    ln2_hi, ln2_lo = split(ln2)
    inv = float(256 / ln2)

    def coarse(v):
        hi = float((v * 2**42).to_integral_value()) / 2**42
        return hi, float(v - Decimal(hi))

    flog = []
    for i in range(256):
        c = Decimal(1) if i == 0 else Decimal(2) if i == 255 else 1 + (Decimal(i) + Decimal("0.5")) / 256
        rc = float(1 / c)
        hi, lo = coarse(-Decimal(rc).ln() - (ln2 if i >= 106 else 0))
        flog.append((rc, hi, lo))
    fln2 = coarse(ln2)

    def row(pairs):
        return ",\n".join("  %s, %s" % (a.hex(), b.hex()) for a, b in pairs)

    out = []
    out.append("/* hg_pow_tables.h -- generated by gen_pow_tables.py; do not edit.")
    out.append(" * Double-double tables of hg_crpow.h (hi, lo pairs, decimal module at 80 digits). */")
    out.append("#ifndef HG_POW_TABLES_H")
    out.append("#define HG_POW_TABLES_H")
    out.append("#define HG_POW_K0 %d       /* LOGC index of k = 0 */" % (-K_LO))
    out.append("#define HG_POW_NLOGC %d" % (K_HI - K_LO + 1))
    out.append("#define HG_POW_LN2_HI %s" % ln2_hi.hex())
    out.append("#define HG_POW_LN2_LO %s" % ln2_lo.hex())
    out.append("#define HG_POW_C1 %s       /* log(2)/256, 32 significant bits */" % c1.hex())
    out.append("#define HG_POW_C2 %s" % c2.hex())
    out.append("#define HG_POW_C3 %s" % c3.hex())
    out.append("#define HG_POW_INV_LN2_256 %s" % inv.hex())
    for name, v in (("THIRD", Decimal(1) / 3), ("SIXTH", Decimal(1) / 6)):
        hi, lo = split(v)
        out.append("#define HG_POW_%s_HI %s" % (name, hi.hex()))
        out.append("#define HG_POW_%s_LO %s" % (name, lo.hex()))
    for d in (5, 7, 9, 11, 24, 120, 720, 5040, 40320):
        out.append("#define HG_POW_INV%d %s" % (d, float(Decimal(1) / d).hex()))
    for d in (3, 4, 6, 8):
        out.append("#define HG_POW_INV%d %s" % (d, float(Decimal(1) / d).hex()))
    out.append("#define HG_POW_FLN2_HI %s" % fln2[0].hex())
    out.append("#define HG_POW_FLN2_LO %s" % fln2[1].hex())
    out.append("/* log(1 + k/256), k = %d .. %d */" % (K_LO, K_HI))
    out.append("#define HG_POW_LOGC_TABLE {\\")
    out.append(row(logc).replace("\n", "\\\n") + "}")
    out.append("/* 2^(j/256), j = 0 .. 255 */")
    out.append("#define HG_POW_EXP2_TABLE {\\")
    out.append(row(exp2).replace("\n", "\\\n") + "}")
    out.append("/* quick log: 1/c, -log(1/c) hi and lo, 0 */")
    out.append("#define HG_POW_FLOG_TABLE {\\")
    out.append(",\\\n".join("  %s, %s, %s, 0.0" % (a.hex(), b.hex(), c.hex()) for a, b, c in flog) + "}")
    out.append("#endif")
    with open(os.path.join(HERE, "hg_pow_tables.h"), "w") as f:
        f.write("\n".join(out) + "\n")


if __name__ == "__main__":
    main()
