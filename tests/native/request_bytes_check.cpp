// Host check (built and run by tests/test_request_bytes.py) of the serving loop's memory estimate: what a
// region takes in a batch's arena, planned with the shortest runs, and in the realignment scratch, two
// alignments of a stripe width to a warp, stays below it.
#include <cstdio>
#include <random>
#include <string>

#include "phmm_plan.h"
#include "phmm_sw.h"

using namespace phmm;

int main()
{
    for (int seed = 0; seed < 300; ++seed) {
        std::mt19937_64 rng(seed);
        auto draw = [&](int lo, int hi) { return lo + (int)(rng() % (uint64_t)(hi - lo + 1)); };
        uint32_t nh = (uint32_t)draw(1, seed % 5 ? 40 : 300), nr = (uint32_t)draw(1, 200);
        std::vector<uint64_t> ho{0}, ro{0};
        std::vector<uint32_t> cols;
        uint32_t longest = 0;
        for (uint32_t h = 0; h < nh; ++h) {
            const uint32_t n = (uint32_t)draw(1, seed % 3 ? 300 : 30);
            longest = std::max(longest, n);
            ho.push_back(ho.back() + n);
        }
        for (uint32_t r = 0; r < nr; ++r) {
            cols.push_back((uint32_t)draw(1, seed % 4 ? 250 : 768));
            ro.push_back(ro.back() + cols.back());
        }
        std::vector<uint8_t> hb(ho.back(), 'A'), rb(ro.back(), 'C'), q(rb.size(), 30), gap(rb.size(), 45);
        for (auto& b : hb) b = draw(0, 200) ? 'A' : 'N';
        for (auto& b : rb) b = draw(0, 200) ? 'C' : 'N';
        for (size_t k = 0; k < gap.size(); k += (size_t)draw(20, 2000)) gap[k] = 40;
        const phmm_batch b{1, &nh, &nr, hb.data(), ho.data(), rb.data(), q.data(), gap.data(), gap.data(), q.data(), ro.data()};
        PlanLimits lim;
        lim.max_stream_single = lim.max_stream_multi = 1;
        Plan p;
        std::string err;
        if (build_plan(b, lim, p, err) != PHMM_OK) return 1;
        const uint64_t need = 5 * p.read_bases + 9 * p.hap_bases + p.out_total * (8 + 8 + 1) +
                              p.rerun_slots * sizeof(RerunEntry) + p.items.size() * sizeof(WorkItem) + p.n_reads * 11ull +
                              p.n_haps * 9ull + sizeof(RegionDesc);
        const uint64_t said = region_bytes(p.read_bases, p.hap_bases, p.out_total, p.n_reads, p.n_haps);
        if (need > said || said > 2 * need + 8192) {
            std::printf("seed %d: need %llu, estimate %llu\n", seed, (unsigned long long)need, (unsigned long long)said);
            return 2;
        }
        uint64_t scratch = 0;
        for (int c = 0; c < kSwWrapClass; ++c) {
            uint64_t n = 0;
            for (uint32_t k : cols) n += k <= 32u * (uint32_t)kSwK[c] && (c == 0 || k > 32u * (uint32_t)kSwK[c - 1]);
            scratch += (n + 1) / 2 * sw16_layout(longest, kSwK[c]).total;
        }
        if (realign_scratch_bytes(longest, nr, [&](uint32_t k) { return cols[k]; }) != scratch) return 3;
    }
    std::puts("ok");
    return 0;
}
