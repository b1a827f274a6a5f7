// Host side of the micro-op marks (micro_ops.h).
#include "micro_ops.h"

#include <algorithm>
#include <vector>

namespace frep {

using namespace micro;

void mark_tape(const uint64_t* in, uint32_t n, uint32_t slots, uint64_t* out) {
    constexpr uint32_t NONE = 0xFFFFFFFFu, MANY = 0xFFFFFFFEu;
    std::vector<uint32_t> def(std::max<uint32_t>(slots, 4), NONE);  // the instruction that wrote the slot last
    std::vector<uint32_t> reader(n, NONE);  // the only instruction that reads this one's result, or MANY
    auto read = [&](uint32_t slot, uint32_t by) {
        const uint32_t d = def[slot];
        if (d == NONE) return;  // an input
        if (reader[d] == NONE) reader[d] = by;
        else if (reader[d] != by) reader[d] = MANY;
    };
    for (uint32_t i = 0; i < n; i++) {
        const uint64_t w = in[i];
        const uint32_t op = mo_op(w);
        if (op != M_CONST) read(mo_a(w), i);
        if (mo_binary(op)) read(mo_b(w), i);
        def[mo_out(w)] = i;
    }
    if (n && def[0] != NONE) reader[def[0]] = MANY;  // slot 0 is the result
    auto folds = [&](uint32_t i) {
        if (i + 1 >= n || mo_op(in[i]) != M_CONST || reader[i] != i + 1) return false;
        const uint64_t w = in[i + 1];
        return mo_binary(mo_op(w)) && (mo_a(w) == mo_out(in[i])) != (mo_b(w) == mo_out(in[i]));
    };
    for (uint32_t i = 0; i < n; i++) {
        uint64_t mark = reader[i] < MANY ? MARK_ONE : 0ull;
        if (folds(i)) {
            mark |= MARK_FOLD;
        } else {
            uint32_t j = i + 1;
            if (j < n && folds(j)) j++;  // (its reader is no constant)
            if (j < n && reader[i] == j) mark |= MARK_TEMP;
        }
        out[i] = (in[i] & ~MARKS) | mark;
    }
}

void strip_marks(uint64_t* pool, uint64_t n, uint32_t align) {
    uint64_t at = 0;
    while (at < n) {
        const uint64_t count = pool[at];
        if (count >= 1ull << 32) return;  // past the last record written
        const uint64_t end = std::min(n, at + 1 + count);
        for (uint64_t i = at + 1; i < end; i++) pool[i] &= ~MARKS;
        at += (1 + count + align - 1) / align * align;
    }
}

}  // namespace frep
