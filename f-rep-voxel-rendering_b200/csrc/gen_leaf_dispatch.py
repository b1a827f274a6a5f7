"""Writes leaf_dispatch.cuh: the last-level pass's inner loop over micro-ops
(micro_ops.h) as inline PTX with a jump table (brx.idx), for 2 and 4 cells per
lane.

There is a case per (opcode, operand kinds, store or not), so a case holds
only the loads, the constant and the store that its micro-op needs. All cases
share one indexed branch: with one of its own at the end of each case every
branch got its own copy of the table, past the constant bank's 64 KB, and the
loop took twice the cycles (276 against 145 per micro-op). The next micro-op's
words are loaded inside the case, after its own have been used, so that the
operand loads and the arithmetic cover their latency; the micro-op after the
last one ends the loop, so no case counts. Cells are handled in pairs with the
packed float operations (add / sub / mul .f32x2, each half rounded to nearest
as on its own).

A slot row holds its cells as lds_k / sts_k lay them out: 8 or 16 bytes per
lane. Arithmetic is pt_exec's
(voxelizer.cu), operation for operation. DIV, SIN, COS, EXP and SQRT of a row
(whose expansions would crowd the instruction cache), and the end, leave the
loop: the caller runs that micro-op in C++ and calls again.

    python gen_leaf_dispatch.py   (from this directory; the output is committed)
"""
from pathlib import Path

OPS = {"CONST": 0, "SIN": 1, "COS": 2, "ADD": 3, "SUB": 4, "MUL": 5, "DIV": 6, "MIN": 7, "MAX": 8,
       "EXP": 9, "NEG": 10, "SQRT": 11, "COPY": 12, "END": 13}
KINDS = "SFI"  # operand kinds: slot row, forwarded, constant
SOURCES = ["SS", "FS", "SF", "FF", "SI", "FI", "IS", "IF"]
COMMUTATIVE = ("ADD", "MUL")  # decode_word and decode_single put F before S and I last
BINARY = ("ADD", "SUB", "MUL", "MIN", "MAX")
UNARY = ("NEG", "COPY", "SQRT")
TABLE = 2 * 256
WIDTHS = (2, 4)  # cells per lane


def case_name(idx):
    """The label of dispatch index `idx` (kinds of a and b | op << 4 | no store << 8)."""
    ka, kb, op, ns = idx & 3, idx >> 2 & 3, idx >> 4 & 15, idx >> 8
    name = next((n for n, v in OPS.items() if v == op), None)
    if ka == 3 or kb == 3:
        return "$FRL_EXIT"
    src = KINDS[ka] + KINDS[kb]
    if name == "CONST":
        return f"$FRL_CONST_{ns}" if src == "SS" else "$FRL_EXIT"
    if name in BINARY and src != "II":
        if name in COMMUTATIVE and src in ("SF", "IS", "IF"):
            return "$FRL_EXIT"
        return f"$FRL_{name}_{src}_{ns}"
    if name in UNARY and (src == "FS" or src == "SS" and name != "SQRT"):
        return f"$FRL_{name}_{src[0]}_{ns}"
    return "$FRL_EXIT"


def gen(K):
    P = K // 2  # pairs
    pairs = range(P)
    L = []

    def load(p, off):
        if K == 2:
            return [f"add.u32 %%ad, %%lb, {off};", f"ld.shared.b64 %%{p}0, [%%ad];"]
        return [f"add.u32 %%ad, %%lb, {off};", f"ld.shared.v2.b64 {{%%{p}0, %%{p}1}}, [%%ad];"]

    def store():
        if K == 2:
            return ["st.shared.b64 [%%wa], %%q0;"]
        return ["st.shared.v2.b64 [%%wa], {%%q0, %%q1};"]

    fetch = ["add.u32 %%da, %%da, 16;", "ld.shared.v4.u32 {%%y, %%z, %%w, %%x}, [%%da];"]

    def select(op, i, a, b):
        """min_sel: (b < a) ? b : a; max_sel: (a < b) ? b : a, per half."""
        out = [f"mov.b64 {{%%e0, %%e1}}, {a};", f"mov.b64 {{%%f0, %%f1}}, {b};"]
        for h in (0, 1):
            x, y = (f"%%f{h}", f"%%e{h}") if op == "MIN" else (f"%%e{h}", f"%%f{h}")
            out += [f"setp.lt.f32 %%p, {x}, {y};", f"selp.f32 %%e{h}, %%f{h}, %%e{h}, %%p;"]
        return out + [f"mov.b64 %%q{i}, {{%%e0, %%e1}};"]

    def arith(op, i, a, b):
        if op in ("ADD", "SUB", "MUL"):
            return [f"{op.lower()}.rn.f32x2 %%q{i}, {a}, {b};"]
        if op in ("MIN", "MAX"):
            return select(op, i, a, b)
        if op == "COPY":
            return [f"mov.b64 %%q{i}, {a};"]
        f = {"NEG": "neg.f32", "SQRT": "sqrt.rn.f32"}[op]
        return [f"mov.b64 {{%%e0, %%e1}}, {a};", f"{f} %%e0, %%e0;", f"{f} %%e1, %%e1;",
                f"mov.b64 %%q{i}, {{%%e0, %%e1}};"]

    def finish(ns):
        return ["bra.uni $FRL_NEXT;" if ns else "bra.uni $FRL_STORE;"]

    L += ["{", ".reg .pred %%p;", ".reg .b32 %%lb, %%ad, %%wa, %%da, %%x, %%y, %%z, %%w;",
          ".reg .f32 %%e0, %%e1, %%f0, %%f1;",
          ".reg .b64 " + ", ".join(f"%%{p}{i}" for p in "qab" for i in pairs) + ", %%c;"]
    # operands: %0 = address of the micro-op (in/out), %1..%K = r (in/out), then lane_base
    L += ["mov.b32 %%da, %0;", f"mov.b32 %%lb, %{K + 1};"]
    L += [f"mov.b64 %%q{i}, {{%{1 + 2 * i}, %{2 + 2 * i}}};" for i in pairs]
    L.append("ld.shared.v4.u32 {%%y, %%z, %%w, %%x}, [%%da];")
    L.append("$FRL_TAB: .branchtargets " + ", ".join(case_name(i) for i in range(TABLE)) + ";")
    L.append("bra.uni $FRL_NEXT;")
    for ns in (0, 1):
        addr = [] if ns else ["add.u32 %%wa, %%lb, %%w;"]
        L.append(f"$FRL_CONST_{ns}:")
        L += ["mov.b64 %%c, {%%y, %%y};"] + [f"mov.b64 %%q{i}, %%c;" for i in pairs] + addr + fetch + finish(ns)
        for op in BINARY:
            for src in SOURCES:
                if op in COMMUTATIVE and src in ("SF", "IS", "IF"):
                    continue
                L.append(f"$FRL_{op}_{src}_{ns}:")
                for which, field in ((0, "%%y"), (1, "%%z")):
                    if src[which] == "S":
                        L += load("ab"[which], field)
                    elif src[which] == "I":
                        L.append(f"mov.b64 %%c, {{{field}, {field}}};")
                L += addr + fetch
                for i in pairs:
                    name = {"S": (f"%%a{i}", f"%%b{i}"), "F": (f"%%q{i}", f"%%q{i}"), "I": ("%%c", "%%c")}
                    L += arith(op, i, name[src[0]][0], name[src[1]][1])
                L += finish(ns)
        for op in UNARY:
            for src in ("F" if op == "SQRT" else "SF"):
                L.append(f"$FRL_{op}_{src}_{ns}:")
                if src == "S":
                    L += load("a", "%%y")
                L += addr + fetch
                for i in pairs:
                    L += arith(op, i, f"%%a{i}" if src == "S" else f"%%q{i}", None)
                L += finish(ns)
    L += ["$FRL_STORE:"] + store() + ["$FRL_NEXT:", "brx.idx.uni %%x, $FRL_TAB;"]
    L += ["$FRL_EXIT:", "mov.b32 %0, %%da;"]
    L += [f"mov.b64 {{%{1 + 2 * i}, %{2 + 2 * i}}}, %%q{i};" for i in pairs]
    L.append("}")
    return L


def emit(K):
    outs = ", ".join(['"+r"(at)'] + [f'"+f"(r.v[{i}])' for i in range(K)])
    asm = "\n".join(f'        "{l}\\n\\t"' for l in gen(K))
    return f'''// Runs micro-ops from shared address `at` on {K} cells per lane (slot rows at
// lane_base), the running result in r, up to one that the loop does not run;
// returns that one's address.
__device__ __forceinline__ LeafRun<{K}> leaf_run_{K}(uint32_t at, uint32_t lane_base, FK<{K}> r) {{
    asm volatile(
{asm}
        : {outs}
        : "r"(lane_base)
        : "memory");
    return LeafRun<{K}>{{at, r}};
}}
'''


def text() -> str:
    """The header's contents."""
    head = '''// Generated by gen_leaf_dispatch.py: the last-level pass's loop over micro-ops
// (micro_ops.h) with a jump table (brx.idx). Included by voxelizer.cu after
// FK<K> is defined. A staged micro-op is {y, z, w, x} (operands, output row,
// dispatch index).
#pragma once

template <int K>
struct LeafRun {
    uint32_t at;
    FK<K> r;
};

'''
    return head + "\n".join(emit(k) for k in WIDTHS)


def main():
    out = Path(__file__).with_name("leaf_dispatch.cuh")
    out.write_text(text())
    print("wrote", out)


if __name__ == "__main__":
    main()
