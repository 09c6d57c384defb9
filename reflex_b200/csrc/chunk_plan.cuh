// How a step's rows go through the scratch of the chunked recurrences (chunk_scan.cuh,
// delta_rule_chunk.cu): all chunks of all sequences at once where their scratch is at most about
// 256 MB, else in rounds of `group` sequences by `seg_rows` rows of each, whose scratch is that too.
#pragma once

#include <cuda_runtime.h>

namespace chunk {

struct Plan {
    int seg_rows = 0, n_segs = 0;  // rows of a sequence a round takes; rounds along the rows
    int group = 0;                 // sequences a round takes
    long long places = 0;          // chunks a round has room for
    bool whole = true;             // one round
};

// R rows in n_seq sequences of at most max_rows; chunks of `L` rows, `one` floats of scratch each.
inline Plan plan_rounds(int R, int n_seq, int max_rows, int L, long long one) {
    Plan p;
    if (R <= 0 || n_seq <= 0 || max_rows <= 0 || one <= 0) return p;
    const long long budget = 64LL << 20, most = budget / one > 1 ? budget / one : 1;
    const long long longest = ((long long)max_rows + L - 1) / L, all = (long long)R / L + n_seq;
    long long chunks = longest;
    p.group = n_seq;
    p.places = all;
    if (all > most) {
        // several sequences a round, of each so many chunks that the state's way in and out is little beside them
        const long long few = longest < 8 ? longest : 8, group = most / few > 1 ? most / few : 1;
        p.whole = false;
        if (group < n_seq) p.group = (int)group;
        chunks = most / p.group < longest ? most / p.group : longest;
        p.places = p.group * chunks;
    }
    p.seg_rows = (int)(chunks * L);
    p.n_segs = (int)((longest + chunks - 1) / chunks);
    return p;
}

// A round: sequences seq0 .. seq0 + its grid's share, of each the rows from seg * seg_rows on.
struct Round {
    int seg_rows, seg, seq0, whole;
};
// The place of chunk c (of round r) of sequence `seq`, whose first row of the step is row0.
__device__ __forceinline__ size_t place_in(const Round& r, int L, int row0, int seq, int c) {
    return r.whole ? (size_t)row0 / L + seq + c : (size_t)(seq - r.seq0) * (r.seg_rows / L) + c;
}

}  // namespace chunk
