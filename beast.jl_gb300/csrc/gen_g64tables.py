"""Generate g64tables.h: sin(i pi / 2048) for i = 0..1024 as doubles (round to nearest), the quarter
wave of the 4096-step table of green64.h, and 2 pi / 4096 as a float pair.

Values come from mpmath at 60 digits.
usage: python gen_g64tables.py > g64tables.h
"""
import numpy as np
from mpmath import mp, mpf


def main():
    mp.dps = 60
    c = 2 * mp.pi / 4096
    hi = float(np.float32(float(c)))
    lo = float(np.float32(float(c - mpf(hi))))
    out = ["// generated by gen_g64tables.py -- do not edit", "#pragma once",
           f"#define G64_STEP_HI {np.float32(hi).item():.9e}f", f"#define G64_STEP_LO {np.float32(lo).item():.9e}f",
           "#define G64_SIN_TABLE_INIT { \\"]
    v = [repr(float(mp.sin(i * mp.pi / 2048))) for i in range(1025)]
    v[0], v[1024] = "0.0", "1.0"
    for i in range(0, 1025, 5):
        out.append("  " + ", ".join(v[i:i + 5]) + ("," if i + 5 < 1025 else "") + " \\")
    out.append("}")
    print("\n".join(out))


if __name__ == "__main__":
    main()
