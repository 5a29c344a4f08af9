// Which of a tree's column sizes are transformed together before they are hashed (prover.cpp, commit_evals).
#pragma once
#include <cstddef>

namespace zk {

// A tree's layers are a chain of launches, each of which may start while the one before still runs: a transform between two of them costs some 2 us, and what
// hashing a size early gains, transforms of the next ones written down meanwhile, is nothing for sizes this small. Proofs of 10 columns of 2^6 ... 2^4 rows over three
// trees: 353 us size by size, 343 with groups of 2^13 words; of 7 of 2^10 ... 2^4 rows 448 and 440. With larger groups tall trees wait for their first hash: 100 columns
// of 2^15 ... 2^10 rows over three trees 1,137 us size by size and with 2^13 words, 1,145 with 2^16, 1,158 with 2^17.
constexpr size_t COMMIT_GROUP_WORDS = (size_t)1 << 13;
// words[i]: of the extended columns of a tree's i-th size, tallest first, n >= 1 of them. How many of the first ones are a group.
inline size_t commit_group(const size_t* words, size_t n) {
    size_t k = 1;
    for (size_t sum = words[0]; k < n && sum + words[k] <= COMMIT_GROUP_WORDS; k++) sum += words[k];
    return k;
}

}  // namespace zk
