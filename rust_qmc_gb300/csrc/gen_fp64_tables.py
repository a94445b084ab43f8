"""Tables of the FP64 elementary functions of qmc_fp64.cuh, computed with
mpmath at 40 digits and rounded to doubles (printed as hexadecimal literals):

  kExp2T[j]   2^(j/256), j = 0..255, as a double and what it leaves
  kLogT[i]    (1/c_i, log c_i) for the 128 intervals of z in [0.6875, 1.375)
              that the leading bits of z select; 1/c_i is the rounded
              reciprocal of the interval's midpoint and log c_i is
              -log of that rounded value, so z (1/c_i) - 1 and log c_i belong
              together; the two intervals that meet at 1 have c_i = 1; log c_i
              is rounded to a multiple of 2^-42, as is kLn2Hi, so that
              k kLn2Hi + log c_i is exact
  kLogLo[i]   what that rounding of log c_i leaves; kLn2Lo the same of ln 2
  kSinCosT[j] (cos, sin) of 2 pi j / 256, j = 0..63

Run: python gen_fp64_tables.py > qmc_fp64_tables.cuh"""
import mpmath as mp

mp.mp.dps = 40


def hexd(v):
    return float(v).hex()


def grid(v):
    """v to a multiple of 2^-42."""
    return mp.nint(v * 2 ** 42) / 2 ** 42


def log_rows():
    rows = []
    for i in range(128):
        bits = (0x3fe60000 + (i << 13)) << 32
        lo = mp.mpf(_double(bits))
        hi = mp.mpf(_double(bits + (1 << 45)))
        if i in (79, 80):
            rows.append((mp.mpf(1), mp.mpf(0)))
            continue
        inv = mp.mpf(float(2 / (lo + hi)))
        rows.append((inv, -mp.log(inv)))
    return rows


def _double(bits):
    import struct
    return struct.unpack("<d", struct.pack("<Q", bits))[0]


def table(ctype, name, items, per_line):
    print("__device__ const %s %s[%d] = {" % (ctype, name, len(items)))
    for i in range(0, len(items), per_line):
        print("    " + " ".join(s + "," for s in items[i:i + per_line]))
    print("};")


if __name__ == "__main__":
    print("// Written by gen_fp64_tables.py: tables of the functions of qmc_fp64.cuh.")
    print("#pragma once")
    print("namespace qmc {")
    powers = [mp.mpf(2) ** (mp.mpf(j) / 256) for j in range(256)]
    table("double2", "kExp2T", ["{%s, %s}" % (hexd(v), hexd(v - mp.mpf(float(v)))) for v in powers], 2)
    table("double2", "kLogT", ["{%s, %s}" % (hexd(a), hexd(grid(b))) for a, b in log_rows()], 2)
    table("double", "kLogLo", [hexd(b - grid(b)) for _, b in log_rows()], 4)
    print("constexpr double kLn2Hi = %s, kLn2Lo = %s;" % (hexd(grid(mp.log(2))), hexd(mp.log(2) - grid(mp.log(2)))))
    table("double2", "kSinCosT", ["{%s, %s}" % (hexd(mp.cos(2 * mp.pi * j / 256)), hexd(mp.sin(2 * mp.pi * j / 256)))
                                  for j in range(64)], 2)
    print("}  // namespace qmc")
