// csim_rand.h — the C library's rand() words for randomStabilizerState, made on the
// device (csim_rand.cu).  Not installed.
//
// The generator is r[i] = r[i - 3] + r[i - 31] mod 2^32 (rand() returns the upper 31
// bits), linear over Z / 2^32, so a warp can start anywhere in the sequence:
// x^n mod x^31 - x^28 - 1 holds r[n], r[n + 1], ... as sums of the words before.
// A state's draws have no fixed length (the dimension is drawn first, and vectors are
// drawn until enough are independent), so the states' first words are a chain.  The
// length of a state that starts at a word is computed for every word; then a block per
// segment of the words follows the chains from all words that a state may begin at
// there, and a walk over the segments finds which of them is the true one.
#pragma once

#include <cstdint>

#include "csim_internal.h"

namespace csim {

constexpr int kRawHistory = 34;                  // words in front of a buffer of raw words
constexpr int kRawChunk = 31 * 16;               // words a warp makes
constexpr int kRawJumps = 18;                    // jumps of 2^b chunks
constexpr int64_t kRawMax = (int64_t)kRawChunk << kRawJumps;
constexpr int kMaxSegment = 1 << 16;             // words per segment, at most (16 bits each in shared memory)

struct RawStart {
    uint32_t jump[kRawJumps][31];  // x^(kRawChunk 2^b), coefficient of x^m at m
    uint32_t history[kRawHistory];  // the last words before the buffer's
};
// randomStabilizerState's dimension from a rand() value x: the first d with x <= last[d]
struct DrawTable {
    int n;
    uint32_t last[65];
};
// Where the states of a batch end; device memory
struct DrawChain {
    int64_t states, words;          // states that have their words (fewer if there are not enough), words they take
    uint32_t history[kRawHistory];  // the last words before that point
};

void raw_jumps(RawStart& s);                                // fills jump
void draw_table(int n, const double* cum, DrawTable& t);    // cum: csim_host::cum_table

// words [0, count) of the sequence behind s.history into buf[kRawHistory ...], the history in front
int launch_raw_words(const Launch& L, const RawStart& s, int64_t count, uint32_t* buf);
// Words per segment of the chain of `states` states of up to `longest` words each: a power of two.
// Following a chain within a segment takes 30 ns a state, twice, the walk 300 ns a segment, so
// sqrt(5 states) states per segment are best.
inline int chain_segment(int64_t states, int longest) {
    int64_t s = 1 << 10;
    while (s < kMaxSegment && s * s < 5 * states * longest * longest / 2) s *= 2;
    return (int)s;
}
inline int64_t chain_padded(int64_t count, int segment) { return (count + segment - 1) / segment * segment; }
// len[i] for i < padded (a multiple of 256): the words of a state that starts at word i, 0 if they go
// beyond `count`
int launch_draw_lengths(const Launch& L, const DrawTable& t, const uint32_t* buf, int64_t count, int64_t padded,
                        uint16_t* len);
// offs[0 .. states]: the words that the states begin at (indices into buf) and the end of the last;
// states without enough words get none.  entries: words from a segment's first that most states which
// begin before the segment end by; map: padded / segment * entries words of scratch.
int launch_draw_chain(const Launch& L, const uint16_t* len, int64_t padded, int segment, const uint32_t* buf, int entries,
                      uint32_t* map, int64_t states, int64_t* offs, DrawChain* chain);

}  // namespace csim
