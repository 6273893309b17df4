"""Generate ``exp2_table.h``: 2^(j/512), j = 0..511, rounded to nearest from 60 digits.

The FP64 kernels that have no context to keep an uploaded table in read it (exp64.cuh). Run from
the repository root:

    python inca_parallel_gb300/csrc/gen_exp2.py
"""
import decimal
import os

SIZE = 512


def main():
    decimal.getcontext().prec = 60
    # float() of a decimal string is correctly rounded
    v = [float(decimal.Decimal(2) ** (decimal.Decimal(j) / SIZE)).hex() for j in range(SIZE)]
    out = ["// Generated by gen_exp2.py. Do not edit.",
           f"// 2^(j/{SIZE}), rounded to nearest.",
           "#pragma once",
           "namespace inca {",
           f"static __device__ const double kExp2Table[{SIZE}] = {{"]
    out += ["    " + ", ".join(v[j:j + 4]) + "," for j in range(0, SIZE, 4)]
    out += ["};", "}  // namespace inca"]
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "exp2_table.h")
    with open(path, "w") as f:
        f.write("\n".join(out) + "\n")
    print("wrote", path)


if __name__ == "__main__":
    main()
