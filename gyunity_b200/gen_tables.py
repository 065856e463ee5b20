"""Generate the Sobol' tables header from the reference's table sources.

The Sobol' generator matrices (Joe-Kuo direction numbers as tabulated by
Gruenschloss 2012, reference ``sampler/Sobol.cpp:38``) and the per-pixel
enumeration matrices (``sampler/SobolEnum.cpp:5`` and ``:709``) are data of
the reference. They are not copied into this repository: this script reads
them from a reference checkout and writes ``gyunity_b200/_gen/sobol_tables.h``
(git-ignored). Without a checkout it computes the same numbers: Joe and Kuo's
initial direction numbers from torch's Sobol' engine, extended to 52 columns
by the recurrence of Bratley and Fox (1988), and the enumeration matrices by
inverting dimensions 0 and 1 over GF(2). The built libraries embed the tables,
so machines that only run them need the built ``.so`` files.

Layout of the generated header:
  GYT_SOBOL_DIMS = 1024, GYT_SOBOL_COLS = 52
  static const uint32_t gyt_sobol_matrices[1024 * 52];
  GYT_ENUM_M = number of enumeration levels (max log2 resolution)
  static const uint64_t gyt_vdc_sobol[GYT_ENUM_M][52];
  static const uint64_t gyt_vdc_sobol_inv[GYT_ENUM_M][52];
"""
import hashlib
import os
import re
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
OUT_DIR = os.path.join(HERE, "_gen")
OUT = os.path.join(OUT_DIR, "sobol_tables.h")
HEX = re.compile(r"0x[0-9a-fA-F]+")


def _strip_comments(text):
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _sobol_matrices(path):
    text = _strip_comments(open(path).read())
    start = text.index("Matrices::matrices[")
    body = text[text.index("{", start) + 1:text.index("};", start)]
    vals = [int(h, 16) for h in HEX.findall(body)]
    if len(vals) != 1024 * 52:
        raise RuntimeError("unexpected Sobol matrix count %d" % len(vals))
    return vals


def _jagged(text, name):
    start = text.index(name)
    i = text.index("{", start) + 1
    rows, depth, cur = [], 0, None
    while True:
        ch = text[i]
        if ch == "{":
            depth += 1
            cur = i + 1
        elif ch == "}":
            if depth == 0:
                break
            depth -= 1
            rows.append([int(h, 16) for h in HEX.findall(text[cur:i])])
        i += 1
    return rows


def _enum_tables(path):
    text = _strip_comments(open(path).read())
    fwd = _jagged(text, "vdc_sobol_matrices[]")
    inv = _jagged(text, "vdc_sobol_matrices_inv[]")
    # the inverse table carries one more level than the forward one; only
    # levels present in both are usable (m = log2 of the padded resolution)
    n = min(len(fwd), len(inv))
    fwd, inv = fwd[:n], inv[:n]
    for r in fwd + inv:
        if len(r) > 52:
            raise RuntimeError("enumeration row longer than 52 columns")
    return fwd, inv


def _primitive_polynomials():
    """(degree, coefficient bits) of the primitive polynomials over GF(2) by
    degree, then value: the order in which Joe and Kuo assign them."""
    def is_primitive(poly, deg):
        order = (1 << deg) - 1

        def mul(a, b):
            r = 0
            while b:
                if b & 1:
                    r ^= a
                b >>= 1
                a <<= 1
                if a >> deg & 1:
                    a ^= poly
            return r

        def x_to(e):
            r, b = 1, 2
            while e:
                if e & 1:
                    r = mul(r, b)
                b = mul(b, b)
                e >>= 1
            return r

        primes, f, m = set(), 2, order
        while f * f <= m:
            while m % f == 0:
                primes.add(f)
                m //= f
            f += 1
        if m > 1:
            primes.add(m)
        return x_to(order) == 1 and all(x_to(order // q) != 1 for q in primes)

    yield 1, 3
    deg = 2
    while True:
        for poly in range((1 << deg) + 1, 1 << (deg + 1), 2):
            if is_primitive(poly, deg):
                yield deg, poly
        deg += 1


def _computed_matrices(dims=1024, cols=52):
    """The generator matrices without a checkout. The first columns of every
    dimension come from the points themselves: in Gray-code order, point 2^j
    and its predecessor differ by column j."""
    import torch
    known = 13  # the largest degree among the first 1024 dimensions
    pts = torch.quasirandom.SobolEngine(dims).draw(1 << known, dtype=torch.float64)
    pts = (pts * 2.0 ** 30).to(torch.int64)
    first = [(pts[1 << j] ^ pts[(1 << j) - 1]).tolist() for j in range(known)]
    out = [1 << (31 - j) if j < 32 else 0 for j in range(cols)]  # dimension 0: reversed bits
    polys = _primitive_polynomials()
    for d in range(1, dims):
        deg, poly = next(polys)
        v = [first[j][d] << 2 for j in range(deg)]
        for j in range(deg, cols):
            x = v[j - deg] ^ (v[j - deg] >> deg)
            for k in range(1, deg):
                if poly >> (deg - k) & 1:
                    x ^= v[j - k]
            v.append(x)
        if any(v[j] >> 2 != first[j][d] for j in range(known)):
            raise RuntimeError("Sobol' dimension %d does not follow its recurrence" % d)
        out += v
    return out


def _computed_enum_tables(mats, levels=25, cols=52):
    """The enumeration matrices of 2^m x 2^m films: forward, the pixel
    (x << m | y) that index bit 2m + c reaches; inverse, the low 2m index
    bits of pixel bit c."""
    fwd, inv = [], []
    for m in range(1, levels + 1):
        img = [mats[k] >> (32 - m) << m | mats[cols + k] >> (32 - m) for k in range(cols)]
        basis = {}  # leading bit -> (pixel, the index bits that give it)
        for k in range(2 * m):
            val, comb = img[k], 1 << k
            while val and val.bit_length() - 1 in basis:
                b = basis[val.bit_length() - 1]
                val, comb = val ^ b[0], comb ^ b[1]
            if not val:
                raise RuntimeError("Sobol' dimensions 0 and 1 are dependent at level %d" % m)
            basis[val.bit_length() - 1] = val, comb
        row = []
        for c in range(2 * m):
            val, comb = 1 << c, 0
            while val:
                b = basis[val.bit_length() - 1]
                val, comb = val ^ b[0], comb ^ b[1]
            row.append(comb)
        inv.append(row)
        fwd.append(img[2 * m:])
    return fwd, inv


def generate(reference=None, force=False):
    """Writes the generated header from the reference checkout at
    ``reference`` (else $GYUNITY_REFERENCE); without a checkout an existing
    header is kept, or the tables are computed."""
    reference = reference or os.environ.get("GYUNITY_REFERENCE")
    src = os.path.join(reference, "Gyunity", "src", "sampler") if reference else None
    if os.path.exists(OUT) and not force:
        return OUT
    if src and os.path.isdir(src):
        mats = _sobol_matrices(os.path.join(src, "Sobol.cpp"))
        fwd, inv = _enum_tables(os.path.join(src, "SobolEnum.cpp"))
    else:
        mats = _computed_matrices()
        fwd, inv = _computed_enum_tables(mats)
    os.makedirs(OUT_DIR, exist_ok=True)
    lines = ["// Generated by gyunity_b200/gen_tables.py. Do not edit.",
             "#pragma once", "#include <stdint.h>",
             "#define GYT_SOBOL_DIMS 1024", "#define GYT_SOBOL_COLS 52", "#define GYT_ENUM_M %d" % len(fwd),
             "static const uint32_t gyt_sobol_matrices[GYT_SOBOL_DIMS * GYT_SOBOL_COLS] = {"]
    for k in range(0, len(mats), 8):
        lines.append("  " + ", ".join("0x%08xu" % v for v in mats[k:k + 8]) + ",")
    lines.append("};")
    for nm, tab in (("gyt_vdc_sobol", fwd), ("gyt_vdc_sobol_inv", inv)):
        lines.append("static const uint64_t %s[GYT_ENUM_M][52] = {" % nm)
        for row in tab:
            row = row + [0] * (52 - len(row))
            lines.append("  {" + ", ".join("0x%xull" % v for v in row) + "},")
        lines.append("};")
    data = "\n".join(lines) + "\n"
    digest = hashlib.sha256(data.encode()).hexdigest()[:16]
    data += "#define GYT_TABLES_DIGEST \"%s\"\n" % digest
    with open(OUT, "w") as f:
        f.write(data)
    return OUT


if __name__ == "__main__":
    print(generate(sys.argv[1] if len(sys.argv) > 1 else None, force=True))
