// The work that lbm::monitored_blocks queues, with fakes in place of the GPU:
// a step writes its number into its slot, a copy moves slots to the results.
// Returns LBM_* of the call; out[i] = i + 1 for a result that arrived, counts
// = {steps queued, zeroings, copies}.
#include <cstring>
#include <vector>

#include "lbm_monitor.hpp"

extern "C" int monitored_blocks(uint64_t n, uint64_t block, uint64_t fail_step, uint64_t fail_copy, uint64_t *out,
                                uint64_t *counts)
{
    std::vector<uint64_t> slots(block, ~0ull);
    uint64_t steps = 0, zeroings = 0, copies = 0;
    bool step_failed = false;
    const lbm_status s = lbm::monitored_blocks(
        n, block,
        [&](uint64_t count) {
            if (count > block)
                return LBM_ERR_STATE;
            std::memset(slots.data(), 0, count * sizeof(uint64_t));
            zeroings++;
            return LBM_OK;
        },
        [&](uint64_t slot) {
            if (steps == fail_step) {
                step_failed = true;
                return LBM_ERR_CUDA;
            }
            if (slot >= block || slots[slot] != 0)
                return LBM_ERR_STATE;  // a slot that was not cleared for this step
            slots[slot] = ++steps;
            return LBM_OK;
        },
        [&](uint64_t first, uint64_t count, bool failed) {
            if (failed != step_failed)
                return LBM_ERR_STATE;
            if (copies++ == fail_copy)
                return LBM_ERR_NOMEM;
            if (first + count > n)
                return LBM_ERR_STATE;
            std::memcpy(out + first, slots.data(), count * sizeof(uint64_t));
            return LBM_OK;
        });
    counts[0] = steps;
    counts[1] = zeroings;
    counts[2] = copies;
    return int(s);
}
