// lbm_monitor.hpp -- the order of a monitored call's work, without the GPU.
#pragma once

#include <algorithm>
#include <cstdint>

#include "lbm_b200.h"

namespace lbm {

// n steps in blocks of at most `block`, each with a slot of its own:
//   zero(count)              clears the first `count` slots,
//   step(slot)               queues one step,
//   copy(first, count, err)  queues the copy of the first `count` slots to the
//                            results [first, first + count); err: a step of
//                            this block has failed.
// A step that cannot be queued ends the call with its status; the results of
// the steps queued before it are still copied, as the state has advanced by
// them.
template <typename Zero, typename Step, typename Copy>
lbm_status monitored_blocks(uint64_t n, uint64_t block, Zero zero, Step step, Copy copy)
{
    for (uint64_t first = 0; first < n; first += block) {
        const uint64_t count = std::min(n - first, block);
        lbm_status s = zero(count);
        if (s != LBM_OK)
            return s;
        uint64_t done = 0;
        while (done < count && (s = step(done)) == LBM_OK)
            done++;
        if (done > 0) {
            const lbm_status c = copy(first, done, s != LBM_OK);
            if (s == LBM_OK)
                s = c;
        }
        if (s != LBM_OK)
            return s;
    }
    return LBM_OK;
}

}  // namespace lbm
