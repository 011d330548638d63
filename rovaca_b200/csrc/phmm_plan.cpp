// Batch planner (see phmm_plan.h).
//
// Reference behaviour mirrored here:
//   limits                      src/haplotypecaller/pairhmm/roDV_schedule.cpp:70-73,374-381,445-459
//   pairs with an N go to the   src/haplotypecaller/pairhmm/roDV_schedule.cpp:96,105,417-441
//   intra kernel (N wildcard)   (region API tests 'N' only, :422,:435)
//   empty read or haplotype     src/haplotypecaller/pairhmm/roDV_schedule.cpp:460 (pair skipped,
//                               its likelihood stays NaN, pairhmm_internal.cpp:593)
// Instead of the reference's greedy SIMD grouping (roDV_schedule.cpp:87-142), reads of a region are
// paired (two reads per warp, equal kernel class) and each pair becomes one work item per run of
// the region's haplotypes: the warp streams all of them through both reads.
#include "phmm_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <system_error>
#include <thread>

namespace phmm {

namespace {

bool has_n(const uint8_t* p, uint64_t n) { return n > 0 && std::memchr(p, 'N', (size_t)n) != nullptr; }

// True when every byte equals the first: the array equals itself shifted by one.
bool constant_run(const uint8_t* p, uint64_t n) { return n < 2 || std::memcmp(p, p + 1, (size_t)(n - 1)) == 0; }

struct Run {
    uint16_t lo, hi;
    uint32_t cols;
    uint8_t variant;
};

// Splits haplotypes [0, n) of a region into runs of non-empty haplotypes whose column stream
// stays within max_cols; with split_on_n, a run also never mixes N and non-N haplotypes.
void make_runs(const uint64_t* hoff, const uint8_t* hflags, uint32_t n, uint32_t max_cols, bool split_on_n,
               std::vector<Run>& runs)
{
    runs.clear();
    uint32_t h = 0;
    while (h < n) {
        const uint64_t H = hoff[h + 1] - hoff[h];
        if (H == 0) {
            ++h;
            continue;
        }
        Run r;
        r.lo = (uint16_t)h;
        r.cols = 0;
        r.variant = split_on_n ? (hflags[h] & 1) : kIntra;
        while (h < n) {
            const uint64_t Hh = hoff[h + 1] - hoff[h];
            if (Hh == 0) break;
            if (split_on_n && (hflags[h] & 1) != r.variant) break;
            if (r.cols > 0 && r.cols + Hh > max_cols) break;
            r.cols += (uint32_t)Hh;
            ++h;
        }
        r.hi = (uint16_t)h;
        runs.push_back(r);
    }
}

}  // namespace

TileTable TileTable::defaults()
{
    TileTable t{};
    for (int m = 0; m < kModes32; ++m)
        for (int b = 1; b <= kLenBuckets; ++b) {
            t.kh[m][b - 1] = (uint8_t)std::min(b, kMaxK);
            t.multi[m][b - 1] = b > kMaxK ? 1 : 0;
        }
    return t;
}

bool TileTable::valid(std::string& err) const
{
    for (int m = 0; m < kModes32; ++m)
        for (int b = 1; b <= kLenBuckets; ++b) {
            const int k = kh[m][b - 1];
            const bool mu = multi[m][b - 1] != 0;
            const bool ok = mu ? (k >= kMinMultiKH && k <= kMaxK && k < b) : (k >= b && k <= kMaxK);
            if (!ok) {
                err = "tile shape of mode " + std::to_string(m) + ", bucket " + std::to_string(b) + " (reads of " +
                      std::to_string(32 * (b - 1) + 1) + "-" + std::to_string(32 * b) + " bases): " +
                      (mu ? "multi-stripe" : "single-stripe") + " with " + std::to_string(k) +
                      " row pairs per lane cannot hold it";
                return false;
            }
        }
    return true;
}

// kRunSetupCols: an item's fill and drain (31 columns) and its row set-up, in columns' time.  Measured
// on B200 (one call end to end, milliseconds; runs of up to 8192 columns first, then 24, 96, 160): one
// region of 16 haplotypes and 250 reads 1.16, 0.41, 0.42, 0.40; 8 regions 3.13, 0.94, 0.97, 0.95; 150
// regions with per-base gaps 23.8, 21.5, 21.2, 21.5; 24 regions of long reads 21.0, 15.3, 15.1, 15.3;
// 1,000 regions 104.8, 104.6, 104.9, 104.9; 60 low-quality regions 39.8, 39.9, 39.4, 39.4.
constexpr double kRunSetupCols = 96.0;

uint32_t run_cols_for(uint64_t stream_cols, uint64_t warps)
{
    const double c = std::sqrt((double)stream_cols * kRunSetupCols / (double)std::max<uint64_t>(warps, 1));
    return (uint32_t)std::min<double>(std::max(c, 1.0), PlanLimits().max_stream_single);
}

phmm_status scan_batch(const phmm_batch& b, const PlanLimits& lim, BatchScan& s, std::string& err)
{
    s = BatchScan();
    if (b.n_regions == 0) return PHMM_OK;
    if (!b.n_haps || !b.n_reads || !b.hap_off || !b.read_off) {
        err = "batch: n_haps, n_reads, hap_off and read_off are required";
        return PHMM_ERR_INVALID_ARGUMENT;
    }
    uint64_t nh = 0, nr = 0;
    for (uint32_t r = 0; r < b.n_regions; ++r) {
        nh += b.n_haps[r];
        nr += b.n_reads[r];
        if (b.n_haps[r] > lim.max_haps_per_region) {
            err = "region " + std::to_string(r) + ": " + std::to_string(b.n_haps[r]) + " haplotypes exceeds the limit of " +
                  std::to_string(lim.max_haps_per_region);
            return PHMM_ERR_LIMIT_EXCEEDED;
        }
    }
    if (nh > 0xffffffffull || nr > 0xffffffffull) {
        err = "batch: more than 2^32 haplotypes or reads";
        return PHMM_ERR_INVALID_ARGUMENT;
    }
    s.n_haps = (uint32_t)nh;
    s.n_reads = (uint32_t)nr;
    s.hap_base0 = b.hap_off[0];
    s.read_base0 = b.read_off[0];
    // offsets non-decreasing, lengths within the limits; per region the non-empty pairs and cells
    uint64_t h = 0, r = 0;
    for (uint32_t g = 0; g < b.n_regions; ++g) {
        uint64_t hcols = 0, hnon = 0, rrows = 0, rnon = 0, rstripes = 0;
        for (uint32_t k = 0; k < b.n_haps[g]; ++k, ++h) {
            if (b.hap_off[h + 1] < b.hap_off[h]) {
                err = "hap_off is not non-decreasing at " + std::to_string(h + 1);
                return PHMM_ERR_INVALID_ARGUMENT;
            }
            const uint64_t H = b.hap_off[h + 1] - b.hap_off[h];
            if (H > lim.max_hap_len) {
                err = "haplotype " + std::to_string(h) + " longer than " + std::to_string(lim.max_hap_len);
                return PHMM_ERR_LIMIT_EXCEEDED;
            }
            hcols += H;
            hnon += H > 0;
        }
        for (uint32_t k = 0; k < b.n_reads[g]; ++k, ++r) {
            if (b.read_off[r + 1] < b.read_off[r]) {
                err = "read_off is not non-decreasing at " + std::to_string(r + 1);
                return PHMM_ERR_INVALID_ARGUMENT;
            }
            const uint64_t R = b.read_off[r + 1] - b.read_off[r];
            if (R > lim.max_read_len) {
                err = "read " + std::to_string(r) + " longer than " + std::to_string(lim.max_read_len);
                return PHMM_ERR_LIMIT_EXCEEDED;
            }
            rrows += R;
            rnon += R > 0;
            rstripes += (R + (uint64_t)kWarp * kMaxK - 1) / ((uint64_t)kWarp * kMaxK);
        }
        s.out_total += (uint64_t)b.n_haps[g] * b.n_reads[g];
        s.pairs += hnon * rnon;
        s.cells += hcols * rrows;
        s.stream_cols += hcols * ((rstripes + 1) / 2);
    }
    s.hap_bases = b.hap_off[nh] - s.hap_base0;
    s.read_bases = b.read_off[nr] - s.read_base0;
    const bool gaps_needed = lim.region_api == nullptr;
    if ((s.hap_bases > 0 && !b.hap_bases) ||
        (s.read_bases > 0 && (!b.read_bases || !b.read_qual ||
                              (gaps_needed && (!b.read_ins || !b.read_del || !b.read_gcp))))) {
        err = "batch: sequence or quality pointer is null";
        return PHMM_ERR_INVALID_ARGUMENT;
    }
    return PHMM_OK;
}

phmm_status build_plan(const phmm_batch& b, const PlanLimits& lim, Plan& plan, std::string& err)
{
    plan = Plan();
    plan.classes.assign(kPlanClasses, ClassDesc{});
    plan.tiles = lim.tiles ? *lim.tiles : TileTable::defaults();
    plan.region_api = lim.region_api != nullptr;
    if (lim.tiles && !plan.tiles.valid(err)) return PHMM_ERR_INVALID_ARGUMENT;
    const TileTable& tiles = plan.tiles;
    BatchScan sc;
    const phmm_status st = scan_batch(b, lim, sc, err);
    if (st != PHMM_OK || b.n_regions == 0) return st;
    const uint64_t nh = sc.n_haps, nr = sc.n_reads;
    plan.n_regions = b.n_regions;
    plan.n_haps = sc.n_haps;
    plan.n_reads = sc.n_reads;
    plan.hap_base0 = sc.hap_base0;
    plan.read_base0 = sc.read_base0;
    plan.hap_off.resize(nh + 1);
    plan.read_off.resize(nr + 1);
    for (uint64_t h = 0; h <= nh; ++h) plan.hap_off[h] = b.hap_off[h] - plan.hap_base0;
    for (uint64_t r = 0; r <= nr; ++r) plan.read_off[r] = b.read_off[r] - plan.read_base0;
    plan.hap_bases = sc.hap_bases;
    plan.read_bases = sc.read_bases;
    const uint8_t* hb = b.hap_bases + plan.hap_base0;
    const uint8_t* rb = b.read_bases + plan.read_base0;

    plan.hap_flags.resize(nh);
    plan.read_flags.resize(nr);
    plan.regions.resize(b.n_regions);
    {
        uint64_t out_off = 0;
        uint32_t hap_begin = 0, read_begin = 0;
        for (uint32_t g = 0; g < b.n_regions; ++g) {
            RegionDesc& rd = plan.regions[g];
            rd = RegionDesc{};
            rd.out_off = out_off;
            rd.hap_begin = hap_begin;
            rd.n_haps = b.n_haps[g];
            rd.read_begin = read_begin;
            rd.n_reads = b.n_reads[g];
            if (lim.region_api) {
                rd.api = kRegionApi | ((uint32_t)(lim.region_api[g].pcr & 0xff) << 8);
                rd.min_quality = lim.region_api[g].min_quality;
            }
            out_off += (uint64_t)b.n_haps[g] * b.n_reads[g];
            hap_begin += b.n_haps[g];
            read_begin += b.n_reads[g];
        }
        plan.out_total = out_off;
    }

    // Regions are planned independently on host threads: N flags, gap modes, read pairing and haplotype
    // runs, the work items only counted per (FP32 class, stream-length bucket); the items are then written
    // straight to their places.  (A batch has up to an item per read pair and haplotype, so what an item
    // costs here shows in the calls of small and medium batches: written to a list first and sorted from
    // there, 400 regions of 20 reads and 4 haplotypes took 696 us to plan instead of 349.)
    constexpr int kBuckets = 64;
    constexpr uint32_t kBucketCols = 128;
    struct Group {  // reads of one region with one key, against the same runs
        uint32_t region, key;
        uint32_t read, n_reads;  // in Part::reads
        uint32_t run, n_runs;    // in Part::runs
    };
    struct Part {
        std::vector<Group> groups;
        std::vector<uint32_t> reads;
        std::vector<Run> runs;
        std::vector<uint32_t> count;  // items per key; then, while they are written, the next one's place
        uint64_t rerun_cap[kClasses64] = {};
        uint64_t pairs = 0, cells = 0;
        uint32_t max_multi = 0;
    };
    // a group's item for one run, but for its reads, and its sorting key (longest streams of a class first)
    auto item_of = [](const Group& gr, const Run& run, uint32_t& skey) {
        const bool uniform = ((gr.key >> 21) & 1) == 0, read_n = ((gr.key >> 22) & 1) != 0;
        WorkItem it{};
        it.region = gr.region;
        it.hap_lo = run.lo;
        it.hap_hi = run.hi;
        it.kh = (uint8_t)(gr.key & 0xf);
        it.stripes = (uint8_t)((gr.key >> 4) & 0xffff);
        it.variant = read_n ? (uint8_t)kIntra : run.variant;
        it.pmode = (it.variant == kInter && uniform) ? 0 : 1;
        const int c32 = class32(it.variant, it.pmode, it.kh, ((gr.key >> 20) & 1) != 0);
        skey = (uint32_t)c32 * kBuckets + (kBuckets - 1 - std::min<uint32_t>(run.cols / kBucketCols, kBuckets - 1));
        return it;
    };
    auto plan_range = [&](uint32_t g0, uint32_t g1, Part& part) {
        part.count.assign((size_t)kClasses32 * kBuckets, 0);
        std::vector<Run> runs;
        struct ReadKey {
            uint32_t key;  // (N, gap mode, multi, stripes, kh) packed; reads with equal keys share an item
            uint32_t read;
        };
        std::vector<ReadKey> rk;
        for (uint32_t g = g0; g < g1; ++g) {
            const RegionDesc& rd = plan.regions[g];
            const uint32_t M = rd.n_haps, N = rd.n_reads, hap_begin = rd.hap_begin, read_begin = rd.read_begin;
            for (uint32_t h = hap_begin; h < hap_begin + M; ++h)
                plan.hap_flags[h] = has_n(hb + plan.hap_off[h], plan.hap_off[h + 1] - plan.hap_off[h]);
            const uint64_t* hoff = plan.hap_off.data() + hap_begin;
            const uint8_t* hfl = plan.hap_flags.data() + hap_begin;
            rk.clear();
            for (uint32_t r = 0; r < N; ++r) {
                const uint32_t gr = read_begin + r;
                const uint64_t a = plan.read_off[gr], R = plan.read_off[gr + 1] - a;
                plan.read_flags[gr] = has_n(rb + a, R);
                if (R == 0) continue;
                // Mode 0 (the FP32 kernels' PM_EQ): gap qualities constant along the read, insertion
                // and deletion qualities equal (as qualities & 127, which is what the tables read).
                // Region API: gap-open = insertion = deletion, constant unless a PCR model caps them.
                bool uniform;
                if (lim.region_api) {
                    uniform = lim.region_api[g].pcr == PHMM_PCR_NONE;
                } else {
                    const uint8_t* ib = b.read_ins + plan.read_base0 + a;
                    const uint8_t* db = b.read_del + plan.read_base0 + a;
                    const uint8_t* cb = b.read_gcp + plan.read_base0 + a;
                    uniform = constant_run(ib, R) && constant_run(db, R) && constant_run(cb, R) &&
                              (ib[0] & 127) == (db[0] & 127);
                }
                const uint32_t n_flag = plan.read_flags[gr] & 1;
                const int mode = n_flag ? 2 : (uniform ? 0 : 1);
                const int bucket = len_bucket(R);
                const uint32_t kh = tiles.kh[mode][bucket - 1];
                const bool multi = tiles.multi[mode][bucket - 1] != 0;
                const uint32_t stripes = multi ? (uint32_t)((R + kWarp * kh - 1) / (kWarp * kh)) : 1;
                rk.push_back({(n_flag << 22) | ((uniform ? 0u : 1u) << 21) | ((multi ? 1u : 0u) << 20) | (stripes << 4) | kh,
                              gr});
            }
            std::stable_sort(rk.begin(), rk.end(), [](const ReadKey& x, const ReadKey& y) { return x.key < y.key; });
            // the region's runs, for single- and multi-stripe reads without and with an N, once needed
            uint32_t run_at[4], run_n[4] = {}, next = 0;
            for (size_t k = 0; k < rk.size(); k = next) {
                Group gr{};
                gr.region = g;
                gr.key = rk[k].key;
                gr.read = (uint32_t)part.reads.size();
                for (next = (uint32_t)k; next < rk.size() && rk[next].key == gr.key; ++next) part.reads.push_back(rk[next].read);
                gr.n_reads = next - (uint32_t)k;
                const bool read_n = ((gr.key >> 22) & 1) != 0, multi = ((gr.key >> 20) & 1) != 0;
                const int which = (multi ? 2 : 0) + (read_n ? 1 : 0);
                if (run_n[which] == 0) {
                    make_runs(hoff, hfl, M, multi ? lim.max_stream_multi : lim.max_stream_single, !read_n, runs);
                    run_at[which] = (uint32_t)part.runs.size();
                    run_n[which] = (uint32_t)runs.size();
                    part.runs.insert(part.runs.end(), runs.begin(), runs.end());
                }
                gr.run = run_at[which];
                gr.n_runs = run_n[which];
                if (gr.n_runs == 0) continue;
                part.groups.push_back(gr);
                // items, and haplotypes and columns of the runs per mode
                uint64_t haps[kModes32] = {}, cols = 0, rows = 0;
                for (uint32_t j = 0; j < gr.n_runs; ++j) {
                    const Run& run = part.runs[gr.run + j];
                    uint32_t skey;
                    const WorkItem it = item_of(gr, run, skey);
                    part.count[skey] += (gr.n_reads + 1) / 2;
                    haps[mode32(it.variant, it.pmode)] += run.hi - run.lo;
                    cols += run.cols;
                    if (multi) part.max_multi = std::max(part.max_multi, run.cols);
                }
                // each read's pairs may go to the FP64 class of its own length
                for (uint32_t q = 0; q < gr.n_reads; ++q) {
                    const uint32_t r = part.reads[gr.read + q];
                    const uint64_t R = plan.read_off[r + 1] - plan.read_off[r];
                    rows += R;
                    for (int m = 0; m < kModes32; ++m)
                        if (haps[m]) {
                            part.rerun_cap[class64_for_len(m, R)] += haps[m];
                            part.pairs += haps[m];
                        }
                }
                part.cells += cols * rows;
            }
        }
    };
    // the part's items: pairs of a group's reads in order, each against the group's runs in order
    auto write_items = [&](Part& part) {
        std::vector<WorkItem> tmpl;
        std::vector<uint32_t*> place;
        for (const Group& gr : part.groups) {
            tmpl.resize(gr.n_runs);
            place.resize(gr.n_runs);
            for (uint32_t j = 0; j < gr.n_runs; ++j) {
                uint32_t skey;
                tmpl[j] = item_of(gr, part.runs[gr.run + j], skey);
                place[j] = &part.count[skey];
            }
            const uint32_t* reads = part.reads.data() + gr.read;
            for (uint32_t q = 0; q < gr.n_reads; q += 2) {
                const uint32_t r0 = reads[q], r1 = q + 1 < gr.n_reads ? reads[q + 1] : kNoRead;
                for (uint32_t j = 0; j < gr.n_runs; ++j) {
                    WorkItem& it = plan.items[(*place[j])++];
                    it = tmpl[j];
                    it.read[0] = r0;
                    it.read[1] = r1;
                }
            }
        }
    };
    const uint64_t work = plan.read_bases + plan.hap_bases;
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const unsigned nthreads = (unsigned)std::min<uint64_t>({hw, 32u, b.n_regions, work / (1u << 20) + 1});
    std::vector<Part> parts(nthreads);
    // fn(part) for every part, on threads of their own (here, where no other can start)
    auto for_parts = [&](bool threads, auto fn) {
        std::vector<std::thread> pool;
        pool.reserve(nthreads);
        for (unsigned t2 = 1; t2 < nthreads; ++t2) {
            if (threads) {
                try {
                    pool.emplace_back(fn, t2);
                    continue;
                } catch (const std::system_error&) {
                }
            }
            fn(t2);
        }
        fn(0u);
        for (auto& th : pool) th.join();
    };
    {
        // contiguous region ranges with about equal bases each
        std::vector<uint32_t> cut(nthreads + 1, b.n_regions);
        cut[0] = 0;
        uint64_t acc = 0;
        unsigned t = 1;
        for (uint32_t g = 0; g < b.n_regions && t < nthreads; ++g) {
            const RegionDesc& rd = plan.regions[g];
            acc += plan.read_off[rd.read_begin + rd.n_reads] - plan.read_off[rd.read_begin] +
                   plan.hap_off[rd.hap_begin + rd.n_haps] - plan.hap_off[rd.hap_begin];
            if (acc * nthreads >= work * t) cut[t++] = g + 1;
        }
        for_parts(true, [&](unsigned t2) { plan_range(cut[t2], cut[t2 + 1], parts[t2]); });
    }
    // items in the order of their keys, those of one key in region order (a stable counting sort)
    std::vector<uint32_t> start((size_t)kClasses32 * kBuckets + 1, 0);
    for (size_t i = 0; i + 1 < start.size(); ++i) {
        uint32_t at = start[i];
        for (Part& p : parts) {
            const uint32_t n = p.count[i];
            p.count[i] = at;
            at += n;
        }
        start[i + 1] = at;
    }
    const size_t n_items = start.back();
    for (const Part& p : parts) {
        for (int c = 0; c < kClasses64; ++c) plan.classes[kClasses32 + c].rerun_cap += (uint32_t)p.rerun_cap[c];
        plan.pairs += p.pairs;
        plan.cells += p.cells;
        plan.max_multi_stream = std::max(plan.max_multi_stream, p.max_multi);
    }
    plan.empty_pairs = plan.out_total - plan.pairs;
    plan.items.resize(n_items);
    // (a thread costs about as much as 10,000 items)
    for_parts(n_items >= (1u << 16), [&](unsigned t2) { write_items(parts[t2]); });
    for (int c = 0; c < kClasses32; ++c) {
        ClassDesc& cd = plan.classes[c];
        cd.item_off = start[(size_t)c * kBuckets];
        cd.n_items = start[(size_t)(c + 1) * kBuckets] - cd.item_off;
    }
    uint32_t rerun_off = 0;
    for (int c = kClasses32; c < kPlanClasses; ++c) {
        ClassDesc& cd = plan.classes[c];
        cd.rerun_off = rerun_off;
        rerun_off += cd.rerun_cap;
    }
    for (ClassDesc& cd : plan.classes) cd.claim32 = cd.claim64 = cd.rerun_count = cd.rerun_pairs = 0;
    plan.rerun_slots = rerun_off;
    return PHMM_OK;
}

void all_pair_runs(const Plan& plan, uint32_t max_cols, std::vector<RerunEntry>& all, std::vector<ClassDesc>& cd)
{
    constexpr uint32_t kBuckets = 64, kBucketCols = 128;
    const uint32_t single = std::min(PlanLimits().max_stream_single, max_cols);
    const uint32_t striped = std::min(PlanLimits().max_stream_multi, std::max(max_cols / 2, 1u));
    std::vector<std::vector<RerunEntry>> per((size_t)kClasses64 * kBuckets);
    std::vector<Run> runs[4];  // for single- and multi-stripe reads without and with an N
    for (uint32_t g = 0; g < plan.n_regions; ++g) {
        const RegionDesc& rg = plan.regions[g];
        const uint64_t* hoff = plan.hap_off.data() + rg.hap_begin;
        for (auto& r : runs) r.clear();
        for (uint32_t q = 0; q < rg.n_reads; ++q) {
            const uint32_t r = rg.read_begin + q;
            const uint64_t R = plan.read_off[r + 1] - plan.read_off[r];
            if (R == 0) continue;
            const bool read_n = (plan.read_flags[r] & 1) != 0, multi = R > (uint64_t)kWarp * kMaxK;
            std::vector<Run>& rr = runs[(multi ? 2 : 0) + (read_n ? 1 : 0)];
            if (rr.empty())
                make_runs(hoff, plan.hap_flags.data() + rg.hap_begin, rg.n_haps,
                          multi ? striped : single, !read_n, rr);
            for (const Run& run : rr) {
                RerunEntry e;
                e.out_idx = rg.out_off + (uint64_t)run.lo * rg.n_reads + q;
                e.read = r;
                e.hap = rg.hap_begin + run.lo;
                e.n_haps = (uint32_t)(run.hi - run.lo);
                e.out_stride = rg.n_reads;
                const int c = class64_for_len(run.variant == kIntra ? 2 : 1, R);
                per[(size_t)c * kBuckets + kBuckets - 1 - std::min(run.cols / kBucketCols, kBuckets - 1)].push_back(e);
            }
        }
    }
    all.clear();
    cd.assign(kClasses64, ClassDesc{});
    for (int c = 0; c < kClasses64; ++c) {
        cd[c].rerun_off = (uint32_t)all.size();
        for (uint32_t b = 0; b < kBuckets; ++b) {
            const auto& v = per[(size_t)c * kBuckets + b];
            all.insert(all.end(), v.begin(), v.end());
        }
        cd[c].rerun_cap = cd[c].rerun_count = (uint32_t)all.size() - cd[c].rerun_off;
    }
}

}  // namespace phmm
