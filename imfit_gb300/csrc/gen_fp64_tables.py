"""Generate fp64_tables.cuh: the lookup tables of fp64_math.cuh's exp2 and log2.

Table-driven elementary functions (P. T. P. Tang, ACM TOMS 15 (1989) 144 and
16 (1990) 378): exp2 splits off a multiple of 1/64, log2 a reciprocal of the
leading 7 fraction bits.  Run: ``python imfit_gb300/csrc/gen_fp64_tables.py``.
"""
import os

import mpmath as mp

mp.mp.dps = 60


def rows(vals, per=4):
    return "\n".join("  " + " ".join(f"{v.hex()}," for v in vals[i:i + per]) for i in range(0, len(vals), per))


def main():
    exp_t = [float(mp.mpf(2) ** (mp.mpf(j) / 64)) for j in range(64)]
    rec, hi, lo = [], [], []
    for i in range(128):
        c = float(1 / (1 + (mp.mpf(i) + mp.mpf(1) / 2) / 128))
        full = -mp.log(mp.mpf(c), 2)
        h = mp.nint(full * mp.mpf(2) ** 40) / mp.mpf(2) ** 40  # k + h is exact for |k| < 2^12
        rec.append(c)
        hi.append(float(h))
        lo.append(float(full - h))
    e = [mp.log(2) ** k / mp.factorial(k) for k in range(1, 6)]
    l2 = [(-1) ** (k + 1) / (k * mp.log(2)) for k in range(1, 7)]
    out = f"""// fp64_tables.cuh -- generated by gen_fp64_tables.py (do not edit).
//   kExp2Tab[j]  2^(j/64)
//   kLog2Tab     128 reciprocals c_i = 1 / (1 + (i + 1/2)/128), then -log2 c_i
//                rounded to multiples of 2^-40, then the rests
//   IMFIT_EXP2_COEF  (ln 2)^k / k!, k = 1..5 (Taylor coefficients of 2^r - 1)
//   IMFIT_LOG2_COEF  (-1)^(k+1) / (k ln 2), k = 1..6 (of log2(1 + f))
#pragma once
namespace imfit {{
__device__ const double kExp2Tab[64] = {{
{rows(exp_t)}
}};
__device__ const double kLog2Tab[3 * 128] = {{
{rows(rec)}
{rows(hi)}
{rows(lo)}
}};
}}  // namespace imfit
#define IMFIT_EXP2_COEF {{{", ".join(float(v).hex() for v in e)}}}
#define IMFIT_LOG2_COEF {{{", ".join(float(v).hex() for v in l2)}}}
"""
    with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "fp64_tables.cuh"), "w") as f:
        f.write(out)


if __name__ == "__main__":
    main()
