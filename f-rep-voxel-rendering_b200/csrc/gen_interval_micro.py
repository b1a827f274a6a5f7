"""Writes interval_micro.cuh: the interval passes' forward loop over micro-ops
(micro_ops.h) as inline PTX with a jump table (brx.idx), for both roundings (0
nearest, 1 outward) and 1 or 2 cells per lane.

The loop assumes that no operand is NaN, and shows when that may not hold: s
accumulates result * 0 over every ADD, SUB and MUL, which stays 0 exactly while
all of them are finite (a NaN first arises from an infinity). Then min and max
of bounds are the hardware's minimum and maximum (they equal glm's selects but
for the sign of a zero, which no comparison sees), the four endpoint products of
a square need five and those with a constant four operations. The caller runs
the tape again with iv_exec when s is not 0, or when the tape holds a NaN.

As in leaf_dispatch.cuh there is a case per (opcode, operand kinds, store or
not) and one indexed branch. Bounds of the two cells are kept in pairs, (lo0,
lo1) and (hi0, hi1), for the packed float operations (each half rounded in its
direction as on its own); a slot row holds lo0, lo1, hi0, hi1 per lane, or lo, hi
for one cell. MIN / MAX store their choice ballots as iv_exec does. Other
micro-ops, and the end, leave the loop for the caller.

    python gen_interval_micro.py   (from this directory; the output is committed)
"""
from pathlib import Path

OPS = {"CONST": 0, "SIN": 1, "COS": 2, "ADD": 3, "SUB": 4, "MUL": 5, "DIV": 6, "MIN": 7, "MAX": 8,
       "EXP": 9, "NEG": 10, "SQRT": 11, "COPY": 12, "END": 13}
KINDS = "SFI"  # operand kinds: slot row, forwarded, constant
CASES = {"ADD": ["SS", "FS", "FF", "SI", "FI"], "SUB": ["SS", "FS", "SF", "SI", "FI", "IS", "IF"],
         "MUL": ["SS", "FS", "FF", "SI", "FI"], "MIN": ["SS", "FS", "SF", "FI", "IF"],
         "MAX": ["SS", "FS", "SF", "FI", "IF"], "NEG": ["SS", "FS"], "COPY": ["SS", "FS"], "SQRT": ["FS"],
         "CONST": ["SS"]}
TABLE = 2 * 256


def case_name(idx):
    """The label of dispatch index `idx` (kinds of a and b | op << 4 | no store << 8)."""
    ka, kb, op, ns = idx & 3, idx >> 2 & 3, idx >> 4 & 15, idx >> 8
    name = next((n for n, v in OPS.items() if v == op), None)
    if ka == 3 or kb == 3 or KINDS[ka] + KINDS[kb] not in CASES.get(name, []):
        return "$FIM_EXIT"
    return f"$FIM_{name}_{KINDS[ka]}{KINDS[kb]}_{ns}"


def gen(rnd, KI):
    dn, up = ("rm", "rp") if rnd else ("rn", "rn")
    typ = "f32x2" if KI == 2 else "f32"
    reg = ".b64" if KI == 2 else ".f32"
    cells = range(KI)
    L = ["{", ".reg .pred %%p, %%pf, %%ps, %%lane0, %%st;",
         ".reg .b32 %%lb, %%ad, %%wa, %%da, %%x, %%y, %%z, %%w, %%mm, %%cap, %%ln;",
         ".reg .b32 " + ", ".join(f"%%v{b}_{h}" for b in (0, 1) for h in cells) + ";",
         ".reg .b64 %%mb, %%ma, %%mo;",
         f".reg {reg} %%ql, %%qh, %%al, %%ah, %%bl, %%bh, %%c, %%s, %%zero, %%p0, %%p1, %%p2, %%p3, %%u0, %%u1, %%u2, %%u3;",
         ".reg .f32 " + ", ".join(f"%%{n}{h}" for n in ("e", "f", "g", "h", "r", "t") for h in cells) + ";"]

    def unpack(names, src):
        if KI == 1:
            return [f"mov.f32 %%{names}0, {src};"]
        return [f"mov.b64 {{%%{names}0, %%{names}1}}, {src};"]

    def pack(dst, names):
        if KI == 1:
            return [f"mov.f32 {dst}, %%{names}0;"]
        return [f"mov.b64 {dst}, {{%%{names}0, %%{names}1}};"]

    def load(p, off):
        vec = "ld.shared.v2.b64" if KI == 2 else "ld.shared.v2.f32"
        return [f"add.u32 %%ad, %%lb, {off};", f"{vec} {{%%{p}l, %%{p}h}}, [%%ad];"]

    def const(field):
        return [f"mov.b64 %%c, {{{field}, {field}}};"] if KI == 2 else [f"mov.b32 %%c, {field};"]

    def extremes(dst, op, srcs):
        """dst = the op ("min" / "max") of srcs, per cell."""
        out = []
        for n, s in zip("efgh", srcs):
            out += unpack(n, s)
        for h in cells:
            ns = [f"%%{n}{h}" for n in "efgh"[:len(srcs)]]
            out.append(f"{op}.f32 %%r{h}, {', '.join(ns[:3])};")
            if len(ns) == 4:
                out.append(f"{op}.f32 %%r{h}, %%r{h}, {ns[3]};")
        return out + pack(dst, "r")

    fetch = ["add.u32 %%da, %%da, 16;", "ld.shared.v4.u32 {%%y, %%z, %%w, %%x}, [%%da];"]
    track = [f"fma.rn.{typ} %%s, %%ql, %%zero, %%s;", f"fma.rn.{typ} %%s, %%qh, %%zero, %%s;"]

    def mul(d, a, b, i):
        return f"mul.{d}.{typ} {i}, {a}, {b};"

    def arith(op, src, a, b):
        """a, b: (lo, hi) register names."""
        if op == "ADD":
            return [f"add.{dn}.{typ} %%ql, {a[0]}, {b[0]};", f"add.{up}.{typ} %%qh, {a[1]}, {b[1]};"] + track
        if op == "SUB":  # (through %%p0: an operand may be q itself)
            return [f"sub.{dn}.{typ} %%p0, {a[0]}, {b[1]};", f"sub.{up}.{typ} %%qh, {a[1]}, {b[0]};",
                    f"mov{reg} %%ql, %%p0;"] + track
        if op == "MUL":
            if src == "FF":  # a square
                lows = [(a[0], a[0], "%%p0"), (a[0], a[1], "%%p1"), (a[1], a[1], "%%p2")]
                highs = [(a[0], a[0], "%%u0"), (a[1], a[1], "%%u1")]
            elif src[1] == "I":
                lows = [(a[0], "%%c", "%%p0"), (a[1], "%%c", "%%p1")]
                highs = [(a[0], "%%c", "%%u0"), (a[1], "%%c", "%%u1")]
            else:
                pairs = [(a[0], b[0]), (a[0], b[1]), (a[1], b[0]), (a[1], b[1])]
                lows = [(x, y, f"%%p{i}") for i, (x, y) in enumerate(pairs)]
                highs = [(x, y, f"%%u{i}") for i, (x, y) in enumerate(pairs)]
            out = [mul(dn, x, y, r) for x, y, r in lows] + [mul(up, x, y, r) for x, y, r in highs]
            return (out + extremes("%%ql", "min", [r for _, _, r in lows]) +
                    extremes("%%qh", "max", [r for _, _, r in highs]) + track)
        if op in ("MIN", "MAX"):
            out = unpack("e", a[0]) + unpack("f", a[1]) + unpack("g", b[0]) + unpack("h", b[1])
            for h in cells:  # the choices (iv_exec): bit 0 first may be the result, bit 1 second
                out += [f"setp.lt.f32 %%pf, %%f{h}, %%g{h};", f"setp.lt.f32 %%ps, %%h{h}, %%e{h};",
                        "not.pred %%ps, %%ps;", "or.pred %%ps, %%pf, %%ps;", "not.pred %%pf, %%pf;"]
                first, second = ("%%ps", "%%pf") if op == "MIN" else ("%%pf", "%%ps")
                out += [f"vote.sync.ballot.b32 %%v0_{h}, {first}, -1;", f"vote.sync.ballot.b32 %%v1_{h}, {second}, -1;"]
            f = op.lower()
            for h in cells:
                out += [f"{f}.f32 %%r{h}, %%e{h}, %%g{h};", f"{f}.f32 %%t{h}, %%f{h}, %%h{h};"]
            out += pack("%%ql", "r") + pack("%%qh", "t")
            out += ["setp.lt.and.u32 %%st, %%mm, %%cap, %%lane0;", f"mul.wide.u32 %%mo, %%mm, {8 * KI};",
                    "add.s64 %%ma, %%mb, %%mo;"]
            words = ", ".join(f"%%v0_{h}, %%v1_{h}" for h in cells)
            return out + [f"@%%st st.global.v{2 * KI}.u32 [%%ma], {{{words}}};", "add.u32 %%mm, %%mm, 1;"]
        if op == "NEG":
            z = "neg.f32"
            out = unpack("e", a[0]) + unpack("f", a[1])
            for h in cells:
                out += [f"{z} %%e{h}, %%e{h};", f"{z} %%f{h}, %%f{h};"]
            return out + pack("%%ql", "f") + pack("%%qh", "e")
        if op == "SQRT":
            out = unpack("e", a[0]) + unpack("f", a[1])
            for h in cells:
                out += [f"max.f32 %%e{h}, %%e{h}, 0f00000000;", f"sqrt.{dn}.f32 %%e{h}, %%e{h};",
                        f"max.f32 %%f{h}, %%f{h}, 0f00000000;", f"sqrt.{up}.f32 %%f{h}, %%f{h};"]
            return out + pack("%%ql", "e") + pack("%%qh", "f")
        return [f"mov{reg} %%ql, {a[0]};", f"mov{reg} %%qh, {a[1]};"]  # COPY

    # operands: %0 at, %1 mm, then q (lo then hi), s (in / out); lane_base, mmb, mm_cap
    q = [f"%{2 + i}" for i in range(2 * KI)]
    s = [f"%{2 + 2 * KI + i}" for i in range(KI)]
    base = 2 + 3 * KI
    L += ["mov.b32 %%da, %0;", "mov.b32 %%mm, %1;", f"mov.b32 %%lb, %{base};", f"mov.b64 %%mb, %{base + 1};",
          f"mov.b32 %%cap, %{base + 2};", "mov.u32 %%ln, %%laneid;", "setp.eq.u32 %%lane0, %%ln, 0;"]
    if KI == 2:
        L += [f"mov.b64 %%ql, {{{q[0]}, {q[1]}}};", f"mov.b64 %%qh, {{{q[2]}, {q[3]}}};",
              f"mov.b64 %%s, {{{s[0]}, {s[1]}}};", "mov.b64 %%zero, 0;"]
    else:
        L += [f"mov.f32 %%ql, {q[0]};", f"mov.f32 %%qh, {q[1]};", f"mov.f32 %%s, {s[0]};",
              "mov.f32 %%zero, 0f00000000;"]
    L.append("ld.shared.v4.u32 {%%y, %%z, %%w, %%x}, [%%da];")
    L.append("$FIM_TAB: .branchtargets " + ", ".join(case_name(i) for i in range(TABLE)) + ";")
    L.append("bra.uni $FIM_NEXT;")
    for ns in (0, 1):
        addr = [] if ns else ["add.u32 %%wa, %%lb, %%w;"]
        for op, sources in CASES.items():
            for src in sources:
                L.append(f"$FIM_{op}_{src}_{ns}:")
                if op == "CONST":
                    L += const("%%y") + addr + fetch + [f"mov{reg} %%ql, %%c;", f"mov{reg} %%qh, %%c;"]
                else:
                    binary = op in ("ADD", "SUB", "MUL", "MIN", "MAX")
                    for which, field in ((0, "%%y"), (1, "%%z")) if binary else ((0, "%%y"),):
                        if src[which] == "S":
                            L += load("ab"[which], field)
                        elif src[which] == "I":
                            L += const(field)
                    L += addr + fetch
                    regs = {"F": ("%%ql", "%%qh"), "I": ("%%c", "%%c")}
                    L += arith(op, src, regs.get(src[0], ("%%al", "%%ah")), regs.get(src[1], ("%%bl", "%%bh")))
                L.append("bra.uni $FIM_NEXT;" if ns else "bra.uni $FIM_STORE;")
    st = "st.shared.v2.b64" if KI == 2 else "st.shared.v2.f32"
    L += ["$FIM_STORE:", f"{st} [%%wa], {{%%ql, %%qh}};", "$FIM_NEXT:", "brx.idx.uni %%x, $FIM_TAB;",
          "$FIM_EXIT:", "mov.b32 %0, %%da;", "mov.b32 %1, %%mm;"]
    if KI == 2:
        L += [f"mov.b64 {{{q[0]}, {q[1]}}}, %%ql;", f"mov.b64 {{{q[2]}, {q[3]}}}, %%qh;", f"mov.b64 {{{s[0]}, {s[1]}}}, %%s;"]
    else:
        L += [f"mov.f32 {q[0]}, %%ql;", f"mov.f32 {q[1]}, %%qh;", f"mov.f32 {s[0]}, %%s;"]
    return L + ["}"]


def emit(rnd, KI):
    asm = "\n".join(f'        "{l}\\n\\t"' for l in gen(rnd, KI))
    outs = ", ".join(['"+r"(at)', '"+r"(v.mm)'] + [f'"+f"(v.lo[{h}])' for h in range(KI)] +
                     [f'"+f"(v.hi[{h}])' for h in range(KI)] + [f'"+f"(v.s[{h}])' for h in range(KI)])
    return f'''// {"Outward" if rnd else "Nearest"} rounding, {KI} cell(s) per lane: runs micro-ops from shared address `at`
// (slot rows at lane_base) up to one that the loop does not run; returns that
// one's address. MIN / MAX choices go to mmb[mm], mm counted on.
template <>
__device__ __forceinline__ uint32_t iv_micro_run<{rnd}, {KI}>(uint32_t at, uint32_t lane_base, uint2* mmb, uint32_t mm_cap,
                                                   IvMicro<{KI}>& v) {{
    asm volatile(
{asm}
        : {outs}
        : "r"(lane_base), "l"(mmb), "r"(mm_cap)
        : "memory");
    return at;
}}
'''


def text() -> str:
    """The header's contents."""
    head = '''// Generated by gen_interval_micro.py: the interval passes' forward loop over
// micro-ops (micro_ops.h) with a jump table (brx.idx). Included by voxelizer.cu.
// A staged micro-op is {y, z, w, x} (operands, output row, dispatch index).
#pragma once

// The running result's bounds per cell, the finiteness sum, MIN / MAX so far.
template <int KI>
struct IvMicro {
    float lo[KI], hi[KI], s[KI];
    uint32_t mm;
};

template <int ROUND, int KI>
__device__ __forceinline__ uint32_t iv_micro_run(uint32_t at, uint32_t lane_base, uint2* mmb, uint32_t mm_cap,
                                                 IvMicro<KI>& v);

'''
    return head + "\n".join(emit(r, k) for r in (0, 1) for k in (1, 2))


def main():
    out = Path(__file__).with_name("interval_micro.cuh")
    out.write_text(text())
    print("wrote", out)


if __name__ == "__main__":
    main()
