// Micro-ops of the last-level pass: the mark that the host puts on a root
// tape's words and the per-word steps of the decoder that turns a (shortened)
// marked tape into micro-ops. Plain C++ for both sides, so that a host test runs
// the decoder against plain interpretation.
//
// Why: a leaf's shortened tape computes little of what it holds. On 256 random
// primitives a leaf tape has 145 words on average: 26 % load constants, 20 %
// are MIN/MAX that became COPY, and the blends of decided smooth minima still
// multiply constants. With constants computed while decoding and copies
// dropped, a third of the words is left (158 k micro-ops of 459 k words over
// 900 leaf tapes), and most work on the result of the one before, in registers.
//
// Marks live in bits 8-15 of a word of the device tape pools (the public tape
// formats keep those bits zero; the exports strip them):
//   MARK_ONE   one instruction reads the result, and it is not the tape's result;
//   MARK_FOLD  a CONST whose one reader is the next instruction, a binary one
//              that reads it once;
//   MARK_TEMP  the one reader of the result is the next instruction that is not
//              MARK_FOLD.
// Shortening keeps them true: it only removes instructions, one that survives
// has a reader that uses it, and MIN/MAX that became COPY reads one of its
// operands. So marks are found once, on the root tape.
#pragma once
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define FREP_MO_HD __host__ __device__ __forceinline__
#else
#define FREP_MO_HD inline
#endif

namespace frep {
namespace micro {

constexpr uint64_t MARK_ONE = 1ull << 8, MARK_FOLD = 1ull << 9, MARK_TEMP = 1ull << 10;
constexpr uint64_t MARKS = 0xFF00ull;  // everything an export strips

// Opcodes of the wide encoding (tape words' low byte).
constexpr uint32_t M_CONST = 0, M_SIN = 1, M_COS = 2, M_ADD = 3, M_SUB = 4, M_MUL = 5, M_DIV = 6, M_MIN = 7, M_MAX = 8,
                   M_EXP = 9, M_NEG = 10, M_SQRT = 11, M_COPY = 12;
constexpr uint32_t M_END = 13;  // after the last micro-op of a segment

FREP_MO_HD uint32_t mo_op(uint64_t w) { return (uint32_t)w & 0xFFu; }
FREP_MO_HD uint32_t mo_out(uint64_t w) { return ((uint32_t)w >> 16) & 0xFFFFu; }
FREP_MO_HD uint32_t mo_a(uint64_t w) { return (uint32_t)(w >> 32) & 0xFFFFu; }
FREP_MO_HD uint32_t mo_b(uint64_t w) { return (uint32_t)(w >> 48); }
FREP_MO_HD bool mo_binary(uint32_t op) { return op >= M_ADD && op <= M_MAX; }

// A micro-op packed in 64 bits: dispatch index x (bits 0-8) = kinds of the
// operands (a in bits 0-1, b in bits 2-3) | op << 4 | no store << 8; the slots a,
// b and out (5 bits each from bits 9, 14 and 19); a constant (bits 32-63).
// Kinds: S a slot row, F the previous micro-op's result, I the constant. ADD
// and MUL commute bit for bit, so they have no (S, F), (I, S) and (I, F).
// CONST's value is its constant; unary ops have kind S for b.
constexpr uint32_t KIND_S = 0, KIND_F = 1, KIND_I = 2;
constexpr uint32_t MO_NO_STORE = 1u << 8, MO_X = 0x1FFu;
constexpr uint32_t MO_SLOTS = 32;  // a decoded tape names slots below this
FREP_MO_HD uint32_t mo_kind_a(uint32_t x) { return x & 3u; }
FREP_MO_HD uint32_t mo_kind_b(uint32_t x) { return (x >> 2) & 3u; }
FREP_MO_HD uint32_t mo_x_op(uint32_t x) { return (x >> 4) & 15u; }
FREP_MO_HD uint32_t mo_slot_a(uint32_t lo) { return (lo >> 9) & 31u; }
FREP_MO_HD uint32_t mo_slot_b(uint32_t lo) { return (lo >> 14) & 31u; }
FREP_MO_HD uint32_t mo_slot_out(uint32_t lo) { return (lo >> 19) & 31u; }

FREP_MO_HD float mo_float(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}
FREP_MO_HD uint32_t mo_bits(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
#endif
}

// Turns a marked tape into micro-ops, one word after the other. Slots that hold
// a constant are a bit of `consts` and a value kept by the caller; instructions
// on constants alone are computed here with the point pass's operations (no
// multiply-add contraction on either side; SQRT and the transcendentals stay
// micro-ops with a constant operand). A micro-op is handed out when the
// next one is known: a value that the next one takes in a register and nothing
// else reads is not stored, and a word that only renames it (COPY, or x - 0,
// exact for every x: the residue of a decided smooth minimum) becomes the
// micro-op's output slot.
struct Decoder {
    uint32_t consts = 0;  // slots that hold a constant
    uint32_t rows = 0;    // slots that some micro-op reads or writes as a row
    uint32_t lo = 0, imm = 0;    // the micro-op in hand, without its output
    uint32_t out = MO_SLOTS;     // its output slot (MO_SLOTS: none in hand)
    bool one = false;            // one instruction reads it
    uint32_t value = 0;          // the constant of the last word, when it is one
    bool last_const = false;
};

// value(s): the constant in slot s (any bits when it holds none);
// keep(s, v): slot s holds the constant v; emit(lo, imm): a micro-op. Written
// with selects, not branches: the lanes of a warp each have a tape of their own.
template <class Value, class Keep, class Emit>
FREP_MO_HD void decode_word(Decoder& d, uint64_t w, Value value, Keep keep, Emit emit) {
    const uint32_t wl = (uint32_t)w, hi = (uint32_t)(w >> 32), op = wl & 0xFFu, out = (wl >> 16) & 31u;
    const uint32_t a = hi & 31u, b = (hi >> 16) & 31u, bit = 1u << out;
    const bool bin = mo_binary(op), is_const = op == M_CONST, copy = op == M_COPY, sub = op == M_SUB;
    const bool ca = (d.consts >> a) & 1u, cb = (d.consts >> b) & 1u;
    const uint32_t va = value(a), vb = value(b);
    const float x = mo_float(va), y = mo_float(vb);
    // the value of an instruction on constants
    float r = op == M_MUL ? x * y : (sub ? x - y : x + y);
    r = op == M_MIN ? (y < x ? y : x) : r;
    r = op == M_MAX ? (x < y ? y : x) : r;
    r = copy ? x : (op == M_NEG ? -x : r);
    const bool folds = (ca && (copy || op == M_NEG || (bin && cb))) || is_const;
    if (folds && op == M_DIV) r = x / y;
    const uint32_t v = is_const ? hi : mo_bits(r);
    if (folds) keep(out, v);
    d.last_const = folds;
    d.value = folds ? v : d.value;
    d.consts = folds ? d.consts | bit : d.consts & ~bit;
    // or the micro-op's operands
    const bool fa = !ca && a == d.out, fb = bin && !cb && b == d.out;
    const bool rename = fa && d.one && (copy || (sub && cb && vb == 0u));  // (the value in hand)
    const bool put = !folds && !rename;
    const bool stays = d.one && (fa || fb);
    if (put && d.out != MO_SLOTS) {
        emit(d.lo | d.out << 19 | (stays ? MO_NO_STORE : 0u), d.imm);
        d.rows |= stays ? 0u : 1u << (d.out & 31u);
    }
    const uint32_t ka = ca ? KIND_I : (fa ? KIND_F : KIND_S);
    const uint32_t kb = !bin ? KIND_S : (cb ? KIND_I : (fb ? KIND_F : KIND_S));
    const bool swap = (op == M_ADD || op == M_MUL) && (ka == KIND_I || (ka == KIND_S && kb == KIND_F));
    const uint32_t lo = swap ? kb | ka << 2 | op << 4 | b << 9 | a << 14 : ka | kb << 2 | op << 4 | a << 9 | b << 14;
    d.rows |= put ? (ka == KIND_S ? 1u << a : 0u) | (bin && kb == KIND_S ? 1u << b : 0u) : 0u;
    d.lo = put ? lo : d.lo;
    d.imm = put ? (ca ? va : vb) : d.imm;
    d.out = folds ? d.out : out;
    d.one = folds ? d.one : (wl & (uint32_t)MARK_ONE) != 0;
}
// The same for one word by itself, with what its neighbours tell: the constant
// of the word before it (MARK_FOLD) becomes an operand, the result of the last
// word without that mark is forwarded, MARK_TEMP needs no store. Constants that
// are not the next word's stay micro-ops. A warp decodes a tape so with its
// words spread over the lanes.
//
// Whether word `w` is a COPY that only renames the result of the word before it:
// no micro-op, the one that computes the value writes it to the COPY's slot.
FREP_MO_HD bool elided(uint64_t w, uint32_t prev_lo) {
    return mo_op(w) == M_COPY && (prev_lo & (uint32_t)(MARK_FOLD | MARK_TEMP)) == (uint32_t)MARK_TEMP &&
           mo_a(w) == (prev_lo >> 16);
}
// The micro-op of word `w`, neither MARK_FOLD nor elided. prev_lo, prev_hi: the
// word before it; last_out: the output slot of the last word before it without
// MARK_FOLD (any value that is no slot: none); dest_lo: the last of the elided
// words that follow it, itself without any. *rows |= the slots that it reads or
// writes as rows.
FREP_MO_HD uint64_t decode_single(uint64_t w, uint32_t prev_lo, uint32_t prev_hi, uint32_t last_out, uint32_t dest_lo,
                                  uint32_t* rows) {
    const uint32_t hi = (uint32_t)(w >> 32), op = (uint32_t)w & 0xFFu, out = (dest_lo >> 16) & 31u;
    const uint32_t a = hi & 0xFFFFu, b = hi >> 16, c = (prev_lo & (uint32_t)MARK_FOLD) ? prev_lo >> 16 : ~0u;
    const bool bin = mo_binary(op), temp = (dest_lo & (uint32_t)MARK_TEMP) != 0;
    const uint32_t ka = a == c ? KIND_I : (a == last_out ? KIND_F : KIND_S);
    const uint32_t kb = !bin ? KIND_S : (b == c ? KIND_I : (b == last_out ? KIND_F : KIND_S));
    const uint32_t ns = temp ? MO_NO_STORE : 0u;
    *rows |= temp ? 0u : 1u << out;
    if (op == M_CONST || (!bin && ka == KIND_I))  // a constant, or the COPY of one
        return (uint64_t)(op == M_CONST ? hi : prev_hi) << 32 | M_CONST << 4 | ns | out << 19;
    *rows |= (ka == KIND_S ? 1u << (a & 31u) : 0u) | (bin && kb == KIND_S ? 1u << (b & 31u) : 0u);
    const bool swap = (op == M_ADD || op == M_MUL) && (ka == KIND_I || (ka == KIND_S && kb == KIND_F));
    const uint32_t lo = swap ? kb | ka << 2 | op << 4 | (b & 31u) << 9 | (a & 31u) << 14
                             : ka | kb << 2 | op << 4 | (a & 31u) << 9 | (b & 31u) << 14;
    return (uint64_t)prev_hi << 32 | lo | ns | out << 19;
}

// After the last word, which writes the tape's result.
template <class Emit>
FREP_MO_HD void decode_end(Decoder& d, Emit emit) {
    if (d.last_const) {  // (a value in hand is not read any more)
        d.lo = M_CONST << 4;
        d.imm = d.value;
        d.out = 0;
    }
    d.rows |= 1u << d.out;
    emit(d.lo | d.out << 19, d.imm);
}

}  // namespace micro

// Copies n tape words with their marks set (host; `slots` = 1 + the largest
// slot named, any bound above it will do).
void mark_tape(const uint64_t* in, uint32_t n, uint32_t slots, uint64_t* out);
// Clears the marks of every record in words [0, n) of a tape pool copied from
// the device: records follow one another, each [count][count words] padded to
// `align` words.
void strip_marks(uint64_t* pool, uint64_t n, uint32_t align);

}  // namespace frep
