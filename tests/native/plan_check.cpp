// Host check of the batch planner (built and run by tests/test_plan_items.py).
//   plan_check cover SEED   random regions, with empty sequences, N, long reads and short runs: every pair of a
//                           non-empty read and haplotype is in exactly one work item, the items of a class
//                           lie together, longest streams first and regions in order within 128 columns, and
//                           the class and rerun counts add up; the runs of the all-FP64 check cover every
//                           pair once too, in no more runs than the longest streams need
//   plan_check cost         planning time of one batch cut into one item per read pair and into one per read
//                           pair and haplotype (best of 40, microseconds)
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>

#include "../../rovaca_b200/csrc/phmm_plan.h"

using namespace phmm;

namespace {

struct Batch {
    std::vector<uint32_t> nh, nr;
    std::vector<uint64_t> ho{0}, ro{0};
    std::vector<uint8_t> hb, rb, q, ins, del, gcp;
    phmm_batch c{};
    void finish()
    {
        q.assign(rb.size(), 30);
        ins.resize(rb.size(), 45);
        del.assign(rb.size(), 45);
        gcp.assign(rb.size(), 10);
        c = phmm_batch{(uint32_t)nh.size(), nh.data(), nr.data(), hb.data(), ho.data(), rb.data(),
                       q.data(), ins.data(), del.data(), gcp.data(), ro.data()};
    }
};

int cover(int seed)
{
    std::mt19937_64 rng(seed);
    auto draw = [&](int lo, int hi) { return lo + (int)(rng() % (uint64_t)(hi - lo + 1)); };
    Batch b;
    for (int g = 0, n = draw(1, 60); g < n; ++g) {
        b.nh.push_back(draw(0, 12));
        b.nr.push_back(draw(0, 40));
        for (uint32_t k = 0; k < b.nh.back(); ++k) {
            for (int j = draw(0, 9) ? draw(1, 300) : 0; j > 0; --j) b.hb.push_back(draw(0, 900) ? 'A' : 'N');
            b.ho.push_back(b.hb.size());
        }
        for (uint32_t k = 0; k < b.nr.back(); ++k) {
            for (int j = draw(0, 9) ? draw(1, draw(0, 9) ? 256 : 768) : 0; j > 0; --j) b.rb.push_back(draw(0, 900) ? 'C' : 'N');
            b.ro.push_back(b.rb.size());
        }
    }
    b.ins.assign(b.rb.size(), 45);
    for (size_t k = 0; k < b.ins.size(); k += (size_t)draw(50, 3000)) b.ins[k] = 40;
    b.finish();
    PlanLimits lim;
    lim.max_stream_single = (uint32_t)draw(1, 1200);
    lim.max_stream_multi = (uint32_t)draw(1, 600);
    Plan p;
    std::string err;
    if (build_plan(b.c, lim, p, err) != PHMM_OK) return 1;
    std::vector<uint8_t> seen(p.out_total, 0);
    uint64_t pairs = 0, cells = 0, rerun = 0;
    for (int c = 0; c < kClasses32; ++c) {
        const ClassDesc& cd = p.classes[c];
        uint64_t bucket = ~0ull;
        uint32_t region = 0;
        for (uint32_t k = cd.item_off; k < cd.item_off + cd.n_items; ++k) {
            const WorkItem& it = p.items[k];
            if (class32(it.variant, it.pmode, it.kh, it.stripes > 1) != c) return 2;
            const RegionDesc& rg = p.regions[it.region];
            const uint64_t cols = p.hap_off[rg.hap_begin + it.hap_hi] - p.hap_off[rg.hap_begin + it.hap_lo];
            const uint64_t bk = std::min<uint64_t>(cols / 128, 63);
            if (bk > bucket || (bk == bucket && it.region < region)) return 3;
            bucket = bk;
            region = it.region;
            for (uint32_t r : it.read) {
                if (r == kNoRead) continue;
                if (r < rg.read_begin || r >= rg.read_begin + rg.n_reads) return 4;
                cells += cols * (p.read_off[r + 1] - p.read_off[r]);
                for (uint32_t h = it.hap_lo; h < it.hap_hi; ++h, ++pairs)
                    if (seen[rg.out_off + (uint64_t)h * rg.n_reads + (r - rg.read_begin)]++) return 5;
            }
        }
    }
    for (int c = kClasses32; c < kPlanClasses; ++c) rerun += p.classes[c].rerun_cap;
    for (uint32_t g = 0; g < p.n_regions; ++g) {
        const RegionDesc& rg = p.regions[g];
        for (uint32_t h = 0; h < rg.n_haps; ++h)
            for (uint32_t r = 0; r < rg.n_reads; ++r) {
                const bool full = p.hap_off[rg.hap_begin + h + 1] > p.hap_off[rg.hap_begin + h] &&
                                  p.read_off[rg.read_begin + r + 1] > p.read_off[rg.read_begin + r];
                if (seen[rg.out_off + (uint64_t)h * rg.n_reads + r] != full) return 6;
            }
    }
    std::vector<RerunEntry> all;
    std::vector<ClassDesc> cd;
    all_pair_runs(p, 8192, all, cd);
    std::vector<uint8_t> again(p.out_total, 0);
    uint64_t least = 0;
    for (uint32_t g = 0; g < p.n_regions; ++g) {  // every region fits one stream per N-free stretch here
        const RegionDesc& rg = p.regions[g];
        uint64_t groups = 0;
        int last = -1;
        for (uint32_t h = rg.hap_begin; h < rg.hap_begin + rg.n_haps; ++h) {
            const int kind = p.hap_off[h + 1] == p.hap_off[h] ? -1 : p.hap_flags[h] & 1;
            groups += kind >= 0 && kind != last;
            last = kind;
        }
        least += groups * rg.n_reads;
    }
    if (all.size() > least) return 8;
    for (int c = 0; c < kClasses64; ++c) {
        uint64_t bucket = ~0ull;
        for (uint32_t k = cd[c].rerun_off; k < cd[c].rerun_off + cd[c].rerun_count; ++k) {
            const RerunEntry& e = all[k];
            const uint64_t R = p.read_off[e.read + 1] - p.read_off[e.read];
            const bool n = (p.read_flags[e.read] | p.hap_flags[e.hap]) & 1;
            if (c != class64_for_len(n ? 2 : 1, R)) return 9;
            const uint64_t bk = std::min<uint64_t>((p.hap_off[e.hap + e.n_haps] - p.hap_off[e.hap]) / 128, 63);
            if (bk > bucket) return 10;
            bucket = bk;
            for (uint32_t h = 0; h < e.n_haps; ++h)
                if (again[e.out_idx + (uint64_t)h * e.out_stride]++) return 11;
        }
    }
    if (again != seen) return 12;
    return pairs == p.pairs && cells == p.cells && rerun == pairs && p.empty_pairs == p.out_total - pairs ? 0 : 7;
}

double best_us(const Batch& b, uint32_t cols)
{
    PlanLimits lim;
    lim.max_stream_single = cols;
    double best = 1e30;
    for (int k = 0; k < 40; ++k) {
        Plan p;
        std::string err;
        const auto t = std::chrono::steady_clock::now();
        if (build_plan(b.c, lim, p, err) != PHMM_OK) std::exit(9);
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count() * 1e6);
    }
    return best;
}

}  // namespace

int main(int argc, char** argv)
{
    if (argc == 3 && std::string(argv[1]) == "cover") return cover(std::atoi(argv[2]));
    Batch b;
    for (int g = 0; g < 150; ++g) {
        b.nh.push_back(6);
        b.nr.push_back(40);
        for (int k = 0; k < 6; ++k) b.ho.push_back(b.ho.back() + 200);
        for (int k = 0; k < 40; ++k) b.ro.push_back(b.ro.back() + 33);
    }
    b.hb.assign(b.ho.back(), 'A');
    b.rb.assign(b.ro.back(), 'C');
    b.ins.assign(b.rb.size(), 45);
    b.finish();
    const double whole = best_us(b, 8192), cut = best_us(b, 200);
    std::printf("%.1f %.1f\n", whole, cut);
    return 0;
}
