// Micro-op decoding (csrc/micro_ops.h) against plain interpretation, on the
// host. Reads tapes from a file ([count][words...] u64 each), shortens each
// with random MIN/MAX choices (backward liveness; a decided MIN/MAX becomes a
// COPY, as the level passes write it) after marking its root, decodes the
// result and runs both. Exit code 0: all bits equal.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "micro_ops.h"

using namespace frep;
using namespace frep::micro;

static size_t g_ops = 0;

static float apply(uint32_t op, float a, float b) {
    switch (op) {
        case M_ADD: return a + b;
        case M_SUB: return a - b;
        case M_MUL: return a * b;
        case M_DIV: return a / b;
        case M_MIN: return b < a ? b : a;
        case M_MAX: return a < b ? b : a;
        case M_NEG: return -a;
        case M_SQRT: return std::sqrt(a);
        case M_SIN: return std::sin(a);
        case M_COS: return std::cos(a);
        case M_EXP: return std::exp(a);
        default: return a;
    }
}
static float bits(uint32_t u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

static float plain(const std::vector<uint64_t>& t, std::vector<float> s) {
    for (uint64_t w : t) {
        const uint32_t op = mo_op(w);
        if (op == M_CONST) s[mo_out(w)] = bits((uint32_t)(w >> 32));
        else s[mo_out(w)] = apply(op, s[mo_a(w)], mo_binary(op) ? s[mo_b(w)] : 0.0f);
    }
    return s[0];
}

// The micro-ops of a tape, run one by one. Rows hold only the slots that the
// decoder reports (the others are poisoned).
// single: each word by itself (decode_single), 32 at a time as a warp takes them.
static bool decoded(const std::vector<uint64_t>& t, const std::vector<float>& in, bool single, float* out) {
    std::vector<std::pair<uint32_t, uint32_t>> ops;
    const size_t n = t.size();
    auto lo = [&](size_t i, size_t back) { return i >= back ? (uint32_t)t[i - back] : 0xFFFF0000u; };
    auto gone = [&](size_t i) { return i < n && i % 32 && !(t[i] & MARK_FOLD) && elided(t[i], lo(i, 1)); };
    std::vector<uint32_t> values(MO_SLOTS, 0x7fc77777u);
    auto emit = [&](uint32_t lo, uint32_t imm) { ops.push_back({lo, imm}); };
    Decoder d;
    for (size_t i = 0; single && i < n; i++) {
        if ((t[i] & MARK_FOLD) || gone(i)) continue;
        size_t dest = i;
        while (gone(dest + 1)) dest++;
        const uint32_t p1 = lo(i, 1);
        const uint64_t u = decode_single(t[i], p1, i ? (uint32_t)(t[i - 1] >> 32) : 0, ((p1 & (uint32_t)MARK_FOLD) ? lo(i, 2) : p1) >> 16,
                                         (uint32_t)t[dest], &d.rows);
        emit((uint32_t)u, (uint32_t)(u >> 32));
    }
    if (!single) for (uint64_t w : t)
        decode_word(d, w, [&](uint32_t s) { return values[s]; }, [&](uint32_t s, uint32_t v) { values[s] = v; }, emit);
    if (!single) decode_end(d, emit);
    if (ops.size() > t.size()) return false;
    std::vector<float> rows(MO_SLOTS, bits(0x7fc12345u));
    for (size_t s = 0; s < 4; s++)
        if (d.rows >> s & 1) rows[s] = in[s];
    float r = bits(0x7fc54321u);
    for (auto [lo, imm] : ops) {
        const uint32_t x = lo & MO_X, op = mo_x_op(x), ka = mo_kind_a(x), kb = mo_kind_b(x);
        auto row = [&](uint32_t s) { return d.rows >> s & 1 ? rows[s] : bits(0x7fc99999u); };
        if (ka == 3 || kb == 3 || op > M_COPY) return false;
        if (op == M_CONST) {
            if (ka || kb) return false;
            r = bits(imm);
        } else {
            if ((op == M_ADD || op == M_MUL) && (ka == KIND_I || (ka == KIND_S && kb == KIND_F))) return false;
            const bool folds = op != M_SQRT && op != M_SIN && op != M_COS && op != M_EXP;
            if (folds && !single && ka == KIND_I && (kb == KIND_I || !mo_binary(op))) return false;
            if (!mo_binary(op) && kb) return false;
            const float a = ka == KIND_F ? r : (ka == KIND_I ? bits(imm) : row(mo_slot_a(lo)));
            float b = 0;
            if (mo_binary(op)) b = kb == KIND_F ? r : (kb == KIND_I ? bits(imm) : row(mo_slot_b(lo)));
            r = apply(op, a, b);
        }
        if (!(x & MO_NO_STORE)) {
            if (!(d.rows >> mo_slot_out(lo) & 1)) return false;
            rows[mo_slot_out(lo)] = r;
        }
    }
    g_ops += ops.size();
    *out = r;
    return true;
}

int main(int argc, char** argv) {
    FILE* f = std::fopen(argv[1], "rb");
    if (argc < 2 || !f) return 2;
    std::mt19937 rng(7);
    uint64_t count;
    size_t tapes = 0, words = 0;
    while (std::fread(&count, 8, 1, f) == 1) {
        std::vector<uint64_t> raw(count), root(count);
        if (std::fread(raw.data(), 8, count, f) != count) return 2;
        uint32_t slots = 4;
        for (uint64_t w : raw) {
            slots = std::max(slots, mo_out(w) + 1);
            if (mo_op(w) != M_CONST) slots = std::max(slots, mo_a(w) + 1);
            if (mo_binary(mo_op(w))) slots = std::max(slots, mo_b(w) + 1);
        }
        mark_tape(raw.data(), (uint32_t)count, slots, root.data());
        // a pool of two records gives back the plain words
        std::vector<uint64_t> pool((2 * (1 + count) + 63) / 16 * 16, 0);
        pool[0] = count;
        std::copy(root.begin(), root.end(), pool.begin() + 1);
        const size_t second = (1 + count + 15) / 16 * 16;
        if (second + 1 + count <= pool.size()) {
            pool[second] = count;
            std::copy(root.begin(), root.end(), pool.begin() + second + 1);
        }
        strip_marks(pool.data(), pool.size(), 16);
        if (pool[0] != count || !std::equal(raw.begin(), raw.end(), pool.begin() + 1)) return 3;
        if (second + 1 + count <= pool.size() &&
            (pool[second] != count || !std::equal(raw.begin(), raw.end(), pool.begin() + second + 1))) return 3;
        for (int round = 0; round < 12; round++) {
            std::vector<uint64_t> t;
            if (round == 0) {
                t = root;
            } else {
                std::vector<bool> live(slots, false);
                live[0] = true;
                const uint32_t both = round % 4;  // the share of undecided MIN/MAX
                for (size_t i = count; i-- > 0;) {
                    uint64_t w = root[i];
                    const uint32_t op = mo_op(w);
                    if (!live[mo_out(w)]) continue;
                    live[mo_out(w)] = false;
                    if (op == M_MIN || op == M_MAX) {
                        const uint32_t c = rng() % 4 < both ? 2 : rng() % 2;
                        if (c != 1) live[mo_a(w)] = true;
                        if (c != 0) live[mo_b(w)] = true;
                        if (c == 0) w = (w & ~0xFFull) | M_COPY;
                        if (c == 1) w = (w & ~0xFFull & ~(0xFFFFull << 32)) | M_COPY | ((uint64_t)mo_b(w) << 32);
                    } else if (op != M_CONST) {
                        live[mo_a(w)] = true;
                        if (mo_binary(op)) live[mo_b(w)] = true;
                    }
                    t.push_back(w);
                }
            }
            if (slots > 32) break;
            if (round) std::reverse(t.begin(), t.end());
            for (int k = 0; k < 4; k++) {
                std::vector<float> in(slots, 0.0f);
                for (int i = 0; i < 4; i++) in[i] = std::uniform_real_distribution<float>(-2.0f, 2.0f)(rng);
                float want = plain(t, in), got;
                if (!decoded(t, in, k % 2, &got)) return 4;
                uint32_t x, y;
                std::memcpy(&x, &want, 4);
                std::memcpy(&y, &got, 4);
                if (x != y && !(std::isnan(want) && std::isnan(got))) {
                    std::printf("tape %zu round %d: %a != %a\n", tapes, round, want, got);
                    return 1;
                }
                words += t.size();
            }
        }
        tapes++;
    }
    std::printf("%zu tapes, %zu words, %zu micro-ops\n", tapes, words, g_ops);
    return 0;
}
