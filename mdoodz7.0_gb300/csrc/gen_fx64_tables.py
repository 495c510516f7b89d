"""Generate fx64_tables.inc: the integer tables of fx64.cuh, rounded to nearest from 70-digit
decimal arithmetic.

    python gen_fx64_tables.py > fx64_tables.inc
"""
from decimal import Decimal, getcontext

getcontext().prec = 70
LN2 = Decimal(2).ln()


def fixed(x, bits):
    return int((x * 2 ** bits).to_integral_value())


def sin_cos(x):
    """sin and cos by their Taylor series (x < 2)."""
    s, c, t, n = Decimal(0), Decimal(0), Decimal(1), 0
    while abs(t) > Decimal(10) ** -60:
        sign = -1 if (n // 2) % 2 else 1
        if n % 2:
            s += sign * t
        else:
            c += sign * t
        n += 1
        t = t * x / n
    return s, c


def table(name, entries, per=4):
    rows = [", ".join(entries[i:i + per]) for i in range(0, len(entries), per)]
    print(f"#define {name} {{ \\\n" + ", \\\n".join(rows) + " }")


def main():
    print("// generated by gen_fx64_tables.py -- do not edit")
    table("MDZ_FX_EXP2_TABLE", [f"{fixed((LN2 * j / 256).exp(), 62):#x}ull" for j in range(256)])
    c = [fixed(Decimal(1) / (1 + (j + Decimal("0.5")) / 256), 16) for j in range(256)]
    table("MDZ_FX_C_TABLE", [f"{x}u" for x in c], 12)
    table("MDZ_FX_LOGC_TABLE", [f"{fixed(-(Decimal(x) / 65536).ln(), 64):#x}ull" for x in c])
    pairs = [sin_cos(Decimal(j) / 256) for j in range(384)]
    table("MDZ_FX_SINCOS_TABLE", [f"{{{fixed(s, 63):#x}ull, {fixed(k, 63):#x}ull}}" for s, k in pairs], 2)


if __name__ == "__main__":
    main()
