// Structures shared by the host runtime and the device kernels.
#pragma once
#include <stdint.h>

namespace mkb {

// Comb geometry for the fixed-base multiply.
//
// A clamped scalar is s = 2^254 + 8·m with m = bits 3..253 (251 bits), so
// s·B = 2^254·B + Σ_i d_i · (2^(off_i) · 8B) where d_i are the digits of m.
// Rows 0..rows-2 use signed digits in [-2^(w-1), 2^(w-1)) with a carry into the next
// row; the top row's digit is unsigned in [0, 2^w_top] and its entries include the
// 2^254·B term.  Row i holds entries k·2^(off_i)·8B for k = 0..cols_i-1.
constexpr int MAX_ROWS = 64;  // 63 rows of 4-bit digits at most

struct CombGeom {
    uint32_t rows;
    uint32_t width[MAX_ROWS];
    uint32_t offset[MAX_ROWS];   // bit offset of digit i inside m
    uint64_t row_base[MAX_ROWS]; // first entry of row i
    uint64_t cols[MAX_ROWS];
    uint64_t entries;
};

// Words per table entry: (y+x, y-x, 2dxy) canonical, 8 little-endian u32 each.
constexpr int ENTRY_WORDS = 24;
// Comb-table entries take 128 bytes, -2dxy as the last 32: every gather reads 96 bytes of exactly
// one aligned 128-byte line, with the third coordinate of the digit's sign.
constexpr int COMB_STRIDE_WORDS = 32;

// Matcher: up to MAX_NEEDLES needles tested in one pass.
//   text needles (contains / suffix, fold): bit-parallel shift-and over the 43 searched
//   base64 characters; needle n occupies bits [bit0, bit0+len) of a multi-word state.
//   regex needles: DFA walk over a states×65×u16 table in device memory.
constexpr int MAX_NEEDLES = 128;
constexpr int SA_WORDS = 8;  // shift-and state words (512 bits of concatenated needles)

struct MatchSet {
    uint32_t n_text;              // text needles packed into the shift-and state
    uint32_t n_regex;             // regex needles
    uint32_t sa_words;            // words of shift-and state in use
    uint32_t short_words;         // with gram4: the leading words, holding the needles shorter than 4
                                  // characters, that every key scans; the rest only when gram4 fires
    uint32_t narrow;              // 1: word 0 has its needles in its low 32 bits (all text needles, or with
                                  // gram4 the short ones)
    // shift-and: per word and value v (0..63) the bits of needle positions accepting v.  Word
    // major, so that the 32 lanes' reads of one word at different values spread over the
    // shared-memory banks (value major, a row of 64 bytes put every lane on bank 0 or 16)
    uint64_t mask[SA_WORDS][64];
    uint64_t first_bit[SA_WORDS]; // bit 0 of every text needle (set on each step)
    uint64_t last_bit[SA_WORDS];  // last bit of every contains-needle
    uint64_t suffix_bit[SA_WORDS];// last bit of every suffix-needle (tested at the end only)
    uint16_t text_id[MAX_NEEDLES];// caller's needle index per text needle
    uint16_t text_last[MAX_NEEDLES]; // global bit index of each text needle's last bit
    // quick compare: when every text needle is case-sensitive (or holds no letter) and they are at
    // most QUICK_CONTAINS contains-needles of 3+ characters and QUICK_SUFFIX suffixes, a key is
    // compared as a bit string first: the first 30 bits (5 characters) of a contains-needle, left
    // aligned, at every position, the last 30 of a suffix, right aligned, at the end
    uint32_t quick;               // 1: on
    uint32_t n_quick_contains, n_quick_suffix;
    uint32_t quick_value[6], quick_mask[6];  // the contains-needles, then from QUICK_CONTAINS the suffixes
    // bucket filter: bit 12·k + b of bucket[v] is set when something in bucket b takes value v as its
    // character k (k < 5): a needle that gram4 holds, or a regex on its last way from its start state to
    // a match.  What may end with the key after k < 5 characters has bits 12·k + b and up in
    // bucket_end (a 4-character needle takes every value as its fifth)
    uint32_t buckets;             // 1: on
    uint32_t text_buckets;        // the buckets of needles
    uint64_t bucket[64];
    uint64_t bucket_end;
    uint32_t regex_always;        // the regex needles without a bucket: every key walks their DFAs
    uint32_t n_filtered;          // regex needles with one: filtered[i] has bucket BUCKETS - 1 - i
    uint8_t filtered[16];
    // regex needles
    const uint8_t* dfa[16];
    uint32_t dfa_states[16];
    uint16_t regex_id[16];
    // prefilter of the text needles of 4 or more characters (null: none): bit g of 2^24 is set
    // when some such needle starts with the 4 base64 values g = v0<<18 | v1<<12 | v2<<6 | v3
    // (all case variants of a folded needle)
    const uint32_t* gram4;
};

constexpr uint32_t QUICK_CONTAINS = 2, QUICK_SUFFIX = 4;
constexpr uint32_t BUCKETS = 12, BUCKET_CHARS = 5;
constexpr uint32_t REGEX_BUCKETS = 6;  // at most, beside text needles in the filter
constexpr uint32_t GRAM4_WORDS = 1u << 19;  // 2^24 bits
constexpr uint32_t GRAM4_MIN_NEEDLES = 8;   // long text needles from which a job uses the prefilter

struct HitRecord {
    uint64_t index;
    uint32_t needle;
    uint32_t reserved;
};

// Device-side job state for one launch.
struct JobDevice {
    uint32_t hit_count;     // total hits found (may exceed capacity)
    uint32_t status;        // 0 ok, bit 0: stopped on the stop word
    uint32_t stop;          // host-writable stop word (nonzero stops at the next iteration)
    uint32_t pad;
};

}  // namespace mkb
