// Host check (built and run by tests/test_sw_scratch.py) of an alignment batch's scratch: side by side the
// launch groups' pieces are disjoint, shared they start at one place and take the largest's room; and an
// allocation that fails for the first form is tried again for the second.
#include <cstdio>
#include <vector>

#include "phmm_sw.h"

using namespace phmm;

int main()
{
    SwPlan p;
    uint64_t sum = 0, most = 0;
    for (int g = 0; g < kSwGroups; g += 3) {
        p.need[g] = 1000 + 17 * (uint64_t)((g * 7) % kSwGroups);
        sum += p.need[g];
        most = p.need[g] > most ? p.need[g] : most;
    }
    p.lay_out(true);
    if (!p.concurrent || p.scratch != sum) return 1;
    for (int g = 0; g < kSwGroups; ++g)
        for (int h = 0; h < g; ++h)
            if (p.need[g] && p.need[h] && p.scratch_off[h] + p.need[h] > p.scratch_off[g]) return 2;
    // room for less than the groups side by side
    std::vector<uint64_t> asked;
    uint64_t room = sum - 1;
    auto alloc = [&] {
        asked.push_back(p.scratch);
        return p.scratch <= room ? PHMM_OK : PHMM_ERR_OUT_OF_MEMORY;
    };
    if (sw_alloc(p, alloc) != PHMM_OK || asked != std::vector<uint64_t>{sum, most} || p.concurrent) return 3;
    for (int g = 0; g < kSwGroups; ++g)
        if (p.scratch_off[g] != 0 || p.need[g] > p.scratch) return 4;
    // room for neither; a batch of one group is not tried twice; other errors are not either
    p.lay_out(true);
    room = most - 1;
    asked.clear();
    if (sw_alloc(p, alloc) != PHMM_ERR_OUT_OF_MEMORY || asked.size() != 2) return 5;
    SwPlan one;
    one.need[4] = 500;
    one.lay_out(true);
    int calls = 0;
    if (sw_alloc(one, [&] { return ++calls, PHMM_ERR_OUT_OF_MEMORY; }) != PHMM_ERR_OUT_OF_MEMORY || calls != 1) return 6;
    p.lay_out(true);
    calls = 0;
    if (sw_alloc(p, [&] { return ++calls, PHMM_ERR_CUDA; }) != PHMM_ERR_CUDA || calls != 1 || !p.concurrent) return 7;
    std::puts("ok");
    return 0;
}
