"""Prints the table of normal64.cuh: erfc(a), (2/sqrt(pi)) exp(-a^2) and the
reciprocal of the latter at a = i/32, i = 0..192, each rounded once to the
nearest double from mpmath at 60 digits.

Run: python dbgenzpaper_b200/csrc/normtab_fit.py > dbgenzpaper_b200/csrc/normtab.h
"""
import mpmath as mp

mp.mp.dps = 60


def main():
    print("/* {erfc(a), g(a) = 2/sqrt(pi) exp(-a^2), 1/g(a)}, a = i/32 (normtab_fit.py) */")
    for i in range(193):
        a = mp.mpf(i) / 32
        g = 2 / mp.sqrt(mp.pi) * mp.exp(-a * a)
        print("{%s, %s, %s}," % tuple(float(v).hex() for v in (mp.erfc(a), g, 1 / g)))


if __name__ == "__main__":
    main()
