// size_rules.h -- choices by size that host code makes before a launch: plain
// functions of numbers, so that tests reach sizes that no graph of theirs has.
#pragma once

#include <stdint.h>

inline int pgd_bit_length(uint64_t x) {
    int b = 0;
    while (x) { b++; x >>= 1; }
    return b;
}

// Bits of an id in a packed (row, column) word: ids up to max_id (-1: none), and
// max_id + 1 for the row of what sorts behind every edge.  At most 32: two fit a word.
inline int pgd_id_bits(int64_t max_id) {
    const int b = pgd_bit_length((uint64_t)(max_id + 1));
    return b > 0 ? b : 1;
}
