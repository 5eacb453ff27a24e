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
constexpr int kRawJumps = 20;                    // jumps of 2^b chunks
constexpr int64_t kRawMax = (int64_t)kRawChunk << kRawJumps;
constexpr int kMaxSegment = 1 << 16;             // words per segment, at most (16 bits each in shared memory)

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

// The words of a batch of states from one stream, and the states' places in them
struct DrawJob {
    uint32_t history[kRawHistory];  // the last words before the batch's
    DrawTable table;
    int32_t segment, entries;       // words per segment; words from a segment's first that most states which begin
                                    // before the segment end by
    int64_t words, states;          // words to make
    uint32_t* buf;                  // kRawHistory + words: the history, then the words
    uint16_t* len;                  // padded(): the words of a state that starts at each word (scratch)
    uint32_t* map;                  // map_words() (scratch)
    int64_t* offs;                  // states + 1: the words that the states begin at (indices into buf) and the end of
                                    // the last; states without enough words get none
    DrawChain* chain;
    int64_t padded() const { return (words + segment - 1) / segment * segment; }
    int64_t map_words() const { return padded() / segment * entries; }
};

// Words of the longest sequence for a state of t qubits that draws at most two vectors again
inline int most_words(int t) {
    const int bytes = (t + 7) / 8;
    int most = 0;
    for (int d = 0; d <= t; d++) {
        const int w = 1 + (5 + d) * bytes + (t - d) * (t - d - 1) / 2;
        most = w > most ? w : most;
    }
    return most;
}
// Fills a job but for its history and pointers.  cum: csim_host::cum_table.  Words: `percent` of that
// longest sequence and a few thousand.
void draw_job(int t, const double* cum, int64_t states, int percent, DrawJob& j);

// Four launches for up to kDrawJobs jobs
constexpr int kDrawJobs = 16;
int launch_draws(const Launch& L, const DrawJob* jobs, int njobs);

}  // namespace csim
