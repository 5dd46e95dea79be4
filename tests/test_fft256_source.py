"""The index expressions that csrc/fft256_cluster.cuh itself contains (read from its text, evaluated
here) reproduce the layouts of test_fft256_regions.py: a change of the header that leaves its bank
pattern, its warps' regions or the other side of an exchange behind is seen without a GPU."""
import os
import re

from tests.conftest import ROOT
from tests.test_fft256_regions import AP, BP, GS, LP, ax, bx, lx

TXT = open(os.path.join(ROOT, "quantem_b200", "csrc", "fft256_cluster.cuh")).read()


def _between(start, end):
    a = TXT.index(start)
    return TXT[a: TXT.index(end, a)]


def _expr(text, pattern):
    m = re.search(pattern, text)
    assert m, pattern
    return compile(m.group(1), "fft256_cluster.cuh", "eval")


def _constants():
    env = {}
    for name, value in re.findall(r"\b(GS|LP|BP|AP) = (\d+)", TXT):
        env[name] = int(value)
    return env


def test_constants():
    assert _constants() == {"GS": GS, "LP": LP, "BP": BP, "AP": AP}
    assert "SM_FLOAT2 = 16 * GS" in TXT


def test_line_local_exchange():
    env = _constants()
    base = _expr(TXT, r"local_base\(\) const \{ return (.*?); \}")
    for fn, one, many in (("void line_fwd", "w", "r"), ("void line_bwd", "r", "w")):
        body = _between(fn, "dft_reg<32, INV>(x);\n  }" if fn == "void line_bwd" else "dft8_groups<INV, 0>(x);\n  }")
        at_k1 = _expr(body, rf"float2\* {one} = sm \+ local_base\(\) \+ (tl);")
        off_k1 = _expr(body, rf"\b{one}\[(33 .*?)\]( = x\[k1\]|;)")
        at_g = _expr(body, rf"float2\* {many} = sm \+ local_base\(\) \+ (33 \* tl);")
        off_g = _expr(body, rf"\b{many}\[(8 \* a \+ t)\]")
        for line in range(64):
            b = eval(base, {**env, "line": line})
            for tl in range(8):
                for k1 in range(32):
                    assert b + eval(at_k1, {"tl": tl}) + eval(off_k1, {"k1": k1}) == lx(line, k1, tl)
                for a in range(4):
                    for t in range(8):
                        assert b + eval(at_g, {"tl": tl}) + eval(off_g, {"a": a, "t": t}) == lx(line, 4 * tl + a, t)


def test_slab_exchanges():
    env = _constants()
    a2b, b2a = _between("void a_to_b", "void b_to_a"), _between("void b_to_a", "whole 2-D transforms")
    to_b = _expr(a2b, r"mine = sm \+ (.*?);")
    off_b = _expr(a2b, r"st_peer\(dst \+ 8u \* \(uint32_t\)\((.*?)\), x\[a \* 8 \+ 2 \* d \+ xb\]")
    col = _expr(TXT, r"col_base\(\) const \{ return (.*?); \}")
    assert "float2* r = sm + col_base() + tl;" in a2b and "x[e] = r[8 * e];" in a2b
    to_a = _expr(b2a, r"mine = sm \+ (.*?);")
    pos = _expr(b2a, r"const int pos = (.*?);")
    off_a = _expr(b2a, r"st_peer\(dst \+ 8u \* \(uint32_t\)\((.*?)\), x\[8 \* d \+ j\]")
    row = _expr(TXT, r"row_base\(\) const \{ return (.*?); \}")
    rot = _expr(b2a, r"const int rot = (.*?);")
    assert "float2* r = sm + row_base() + 4 * tl;" in b2a and "float2* ra = r + ((a + rot) & 3);" in b2a
    assert "x[a * 8 + kB] = ra[32 * kB];" in b2a
    for line in range(64):
        for tl in range(8):
            v = {**env, "line": line, "tl": tl}
            for q in range(4):
                w = {**v, "q": q}
                for a in range(4):
                    for xb in range(2):  # register a * 8 + 2 d + xb: column 4 tl + a + 32 (2 d + xb), of rank d
                        assert (eval(to_b, w) + eval(off_b, {**w, "a": a, "xb": xb})
                                == bx(4 * tl + a + 32 * xb, 64 * q + line))
                w["pos"] = eval(pos, w)
                for j in range(8):  # register 8 d + j: row tl + 64 d + 8 j, of rank d
                    assert eval(to_a, w) + eval(off_a, {**w, "j": j}) == ax(tl + 8 * j, 64 * q + line)
            for e in range(32):
                assert eval(col, v) + tl + 8 * e == bx(line, tl + 8 * e)
            for a in range(4):
                for kB in range(8):
                    assert eval(row, v) + 4 * tl + ((a + eval(rot, v)) & 3) + 32 * kB == ax(line, 4 * tl + a + 32 * kB)
