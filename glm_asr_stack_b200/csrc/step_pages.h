// Does a row of a decode batch attend to a token that another row of the same step writes?  (Host only.)
//
// Rows of one batch normally are different sequences with pages of their own.  Two consecutive tokens of one sequence in one
// step, or copies of a sequence that still share the page being filled, are legal too: every layer's cache rows are written
// before any row attends (reference: Infer-engine/cuda/decoder.cu:1972-2139).  The one-launch RoPE + cache write + attention has no
// such order between its CTAs, so these batches take the separate launches.  Decided by whole pages.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "../../include/glmasr_engine_types.h"

namespace glmasr {

// cached[s]: tokens in the cache before this step; every table covers cached[s] + 1 tokens.
inline bool rows_share_new_pages(const glmasr_BlockTable *bts, const int *cached, int n, int block_size) {
    if (n < 2) return false;
    std::vector<int> written((size_t)n);
    uint64_t maybe[64] = {0};               // 4096-bit filter over the written pages: 256 rows x 28 pages cost about 10 us
    for (int s = 0; s < n; ++s) {
        const int b = bts[s].h_table[cached[s] / block_size];
        written[(size_t)s] = b;
        maybe[((unsigned)b >> 6) & 63] |= 1ull << ((unsigned)b & 63);
    }
    std::sort(written.begin(), written.end());
    if (std::adjacent_find(written.begin(), written.end()) != written.end()) return true;
    for (int s = 0; s < n; ++s) {
        const int *t = bts[s].h_table;
        const int own = cached[s] / block_size;
        for (int i = 0; i < own; ++i) {
            const int b = t[i];
            if (((maybe[((unsigned)b >> 6) & 63] >> ((unsigned)b & 63)) & 1) != 0 && std::binary_search(written.begin(), written.end(), b))
                return true;
        }
    }
    return false;
}

}  // namespace glmasr
