"""Emit the lookup tables of the correctly rounded power function
(``hg_crmath.cuh``) as exact hex-float literals, computed with mpmath at
200-bit precision:

* log table: for F_j = 1 + j/1024, j in [LOG_JMIN, LOG_JMAX]:
  RN(1/F_j) and log(F_j) as a double-double (hi, lo);
* exp table: 2^(j/256), j in [0, 256), as a double-double (hi, lo);
* ln 2 split for the exponent term and ln2/256 split for argument reduction;

and those of its integer form (``hg_powint.cuh``), in ``hg_powint_tables.h``:

* r_j = ceil(2^16 / (1 + j/1024)) and round(-log2(r_j / 2^16) 2^64), j in [0, 1024);
* round(2^(j/1024) 2^63), j in [0, 1024);
* the coefficients of both polynomials in fixed point.

Usage: ``python hiten_gb300/csrc/gen_crmath_tables.py`` (needs mpmath).
"""
import os

import mpmath as mp

mp.mp.prec = 200
HERE = os.path.dirname(os.path.abspath(__file__))
LOG_JMIN, LOG_JMAX = -304, 428


def dd(v):
    hi = float(v)
    lo = float(v - mp.mpf(hi))
    return hi, lo


def trunc_bits(v, bits):
    """v rounded toward zero to `bits` significant bits (as a double)."""
    m, e = mp.frexp(v)
    scale = mp.mpf(2) ** bits
    return float(mp.floor(abs(m) * scale) / scale * mp.sign(m) * mp.mpf(2) ** e)


def h(x):
    return float.hex(float(x))


def main():
    out = ["/* Generated by hiten_gb300/csrc/gen_crmath_tables.py (mpmath, 200 bits). */\n",
           "#ifndef HG_CRMATH_TABLES_H\n#define HG_CRMATH_TABLES_H\n\n",
           f"#define HG_LOG_JMIN ({LOG_JMIN})\n#define HG_LOG_JMAX ({LOG_JMAX})\n",
           f"#define HG_LOG_N ({LOG_JMAX - LOG_JMIN + 1})\n\n"]
    inv, lh, ll = [], [], []
    for j in range(LOG_JMIN, LOG_JMAX + 1):
        F = mp.mpf(1) + mp.mpf(j) / 1024
        inv.append(float(1 / F))
        a, b = dd(mp.log(F))
        lh.append(a)
        ll.append(b)
    eh, el = [], []
    for j in range(256):
        a, b = dd(mp.power(2, mp.mpf(j) / 256))
        eh.append(a)
        el.append(b)

    def arr(name, vals):
        body = ",\n  ".join(", ".join(h(v) for v in vals[i:i + 4]) for i in range(0, len(vals), 4))
        return f"#define {name}_INIT {{ \\\n  " + body.replace("\n", " \\\n") + " }\n\n"

    out.append(arr("HG_LOG_INVF", inv))
    out.append(arr("HG_LOG_TH", lh))
    out.append(arr("HG_LOG_TL", ll))
    out.append(arr("HG_EXP_TH", eh))
    out.append(arr("HG_EXP_TL", el))
    ln2 = mp.log(2)
    l2hi = trunc_bits(ln2, 40)
    l2lo = float(ln2 - mp.mpf(l2hi))
    out.append(f"#define HG_LN2_HI {h(l2hi)}\n#define HG_LN2_LO {h(l2lo)}\n")
    c = ln2 / 256
    c1 = trunc_bits(c, 38)
    c2 = trunc_bits(c - mp.mpf(c1), 38)
    c3 = float(c - mp.mpf(c1) - mp.mpf(c2))
    out.append(f"#define HG_L256_1 {h(c1)}\n#define HG_L256_2 {h(c2)}\n#define HG_L256_3 {h(c3)}\n")
    out.append(f"#define HG_INV_L256 {h(256 / ln2)}\n")
    out.append("\n#endif\n")
    with open(os.path.join(HERE, "hg_crmath_tables.h"), "w") as f:
        f.write("".join(out))


def powint():
    r, lg, ex = [], [], []
    for j in range(1024):
        r.append(-(-2**16 * 1024 // (1024 + j)))
        lg.append(int(mp.nint(-mp.log(mp.mpf(r[-1]) / 2**16, 2) * mp.mpf(2)**64)))
        ex.append(int(mp.nint(mp.power(2, mp.mpf(j) / 1024) * mp.mpf(2)**63)))

    def arr(name, vals, fmt):
        return f"#define {name}_INIT {{ \\\n  " + ", \\\n  ".join(
            ", ".join(fmt % v for v in vals[i:i + 4]) for i in range(0, len(vals), 4)) + " }\n\n"

    def fix(name, v, bits, suffix):
        return f"#define {name} {hex(int(mp.nint(v * mp.mpf(2)**bits)))}{suffix}\n"

    a = [None] + [1 / (k * mp.log(2)) for k in range(1, 7)]  # log2(1 + z) = z (a1 - z (a2 - z (a3 - ...)))
    b = [None] + [mp.log(2)**k / mp.factorial(k) for k in range(1, 6)]  # 2^t - 1 = t (b1 + t (b2 + ...))
    out = ["/* Generated by hiten_gb300/csrc/gen_crmath_tables.py (mpmath, 200 bits). */\n",
           "#ifndef HG_POWINT_TABLES_H\n#define HG_POWINT_TABLES_H\n\n",
           arr("HG_PI_R", r, "%d"), arr("HG_PI_L", lg, "0x%016xull"), arr("HG_PI_E", ex, "0x%016xull"),
           fix("HG_PI_A1", a[1] / 2, 64, "ull"), fix("HG_PI_A2", a[2], 64, "ull"), fix("HG_PI_A3", a[3], 33, "u"),
           fix("HG_PI_A4", a[4], 24, "u"), fix("HG_PI_A5", a[5] - a[6] / 2048, 15, "u"),
           fix("HG_PI_B1", b[1], 64, "ull"), fix("HG_PI_B2", b[2], 66, "ull"), fix("HG_PI_B3", b[3], 36, "u"),
           fix("HG_PI_B4", b[4], 26, "u"), fix("HG_PI_B5", b[5], 16, "u"), "\n#endif\n"]
    with open(os.path.join(HERE, "hg_powint_tables.h"), "w") as f:
        f.write("".join(out))


if __name__ == "__main__":
    main()
    powint()
