// Host-side batch planner: validates a phmm_batch, flags reads/haplotypes containing 'N', and cuts
// the batch into wavefront work items grouped by kernel class, longest first inside a class.
#pragma once

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/phmm_b200.h"
#include "phmm_types.h"

namespace phmm {

// Descriptor slots: the FP32 classes, then the FP64 classes (numbering in phmm_types.h).
constexpr int kPlanClasses = kClasses32 + kClasses64;

// FP32 tile shape of every (mode, read-length bucket): kh row pairs per lane, single stripe
// (kh >= bucket) or multi-stripe (kMinMultiKH <= kh < bucket, stripes = ceil(R / (32 * kh))).
// Modes as in phmm_types.h: 0 inter with constant gap qualities (insertion = deletion), 1 inter
// per-row, 2 intra.
struct TileTable {
    uint8_t kh[kModes32][kLenBuckets];
    uint8_t multi[kModes32][kLenBuckets];
    // smallest single stripe up to 256 rows, 256-row stripes beyond
    static TileTable defaults();
    bool valid(std::string& err) const;
};

// Region-API parameters of one region (call_pairhmm semantics): reads arrive with raw base
// qualities and are prepared on the device.
struct RegionApiParams {
    int32_t min_quality;  // base qualities below this become 6
    int32_t pcr;          // phmm_pcr_model
};

struct PlanLimits {
    // Reference limits, roDV_schedule.cpp:70-73 (haplotype index <= 4095, read length <= 768,
    // haplotype length <= 1536).
    uint32_t max_haps_per_region = 4096;
    uint32_t max_read_len = 768;
    uint32_t max_hap_len = 1536;
    // Longest haplotype column stream of one work item (single-stripe reads), and of a
    // multi-stripe item (bounded by the per-warp scratch row).
    uint32_t max_stream_single = 8192;
    uint32_t max_stream_multi = 4096;
    // FP32 tile shapes (null: TileTable::defaults())
    const TileTable* tiles = nullptr;
    // Non-null: every region of the batch uses the region API, with these parameters [n_regions];
    // the batch's gap-quality arrays are not read (the device writes them).
    const RegionApiParams* region_api = nullptr;
};
// a warp's scratch row (24 bytes a column) is read by 16-byte copies, so every row starts on 16 bytes
static_assert(PlanLimits().max_stream_multi % 2 == 0, "scratch rows are not 16-byte aligned");

struct Plan {
    uint32_t n_regions = 0, n_reads = 0, n_haps = 0;
    uint64_t read_bases = 0, hap_bases = 0, out_total = 0;
    uint64_t read_base0 = 0, hap_base0 = 0;  // read_off[0], hap_off[0]: the copy starts there
    uint64_t pairs = 0, cells = 0, empty_pairs = 0;
    std::vector<RegionDesc> regions;
    std::vector<uint64_t> read_off, hap_off;  // rebased to start at 0
    std::vector<uint8_t> read_flags, hap_flags;
    std::vector<WorkItem> items;
    std::vector<ClassDesc> classes;  // kPlanClasses: FP32 classes (items), then FP64 (rerun segments)
    uint64_t rerun_slots = 0;
    uint32_t max_multi_stream = 0;   // longest stream among multi-stripe items (0 if none)
    TileTable tiles{};               // the shapes the items were planned with
    bool region_api = false;         // every region uses the region API (device read prep and post)
    // genotyping events of region-API regions (filled by the caller after planning)
    std::vector<EventDesc> events;
    std::vector<int8_t> hap_allele;
    uint64_t allele_lk_total = 0, gl_total = 0;
};

// Sizes of a batch, from one validating pass over its counts and offsets (no copies).
struct BatchScan {
    uint32_t n_haps = 0, n_reads = 0;
    uint64_t hap_base0 = 0, read_base0 = 0;  // hap_off[0], read_off[0]
    uint64_t hap_bases = 0, read_bases = 0, out_total = 0;
    uint64_t pairs = 0, cells = 0;           // pairs with a non-empty read and haplotype, their cells
    // columns a warp streams over the whole batch: per region its haplotype bases times half its
    // reads (two reads a warp), a read counting once per 256 rows
    uint64_t stream_cols = 0;
};

// The longest haplotype stream of a work item for a batch that streams `stream_cols` columns over
// `warps` resident warps (single-stripe items; multi-stripe items take half).  A long run pays the
// fill, drain and row set-up of an item once for many haplotypes; a short one leaves a small batch
// more items than warps, and a large one a shorter last wave.  With o columns' worth of set-up per
// item the pass takes about (stream_cols (1 + o / c) / warps + c) steps, least at
// c = sqrt(stream_cols o / warps).
uint32_t run_cols_for(uint64_t stream_cols, uint64_t warps);

// Device bytes a region takes in the arena of a batch, at most (the serving loop holds its batches to a
// share of the memory budget by this): gap qualities and bases of the reads, haplotypes with their code
// words, two likelihoods, a flag and a rerun slot per pair, the descriptors, and work items, of which a
// small batch has up to one per read pair and haplotype.
inline uint64_t region_bytes(uint64_t read_bases, uint64_t hap_bases, uint64_t pairs, uint64_t n_reads, uint64_t n_haps)
{
    // (reads pair within one of at most 96 kinds: with or without an N, constant gaps or not, 24 lengths)
    const uint64_t items = (n_reads + std::min<uint64_t>(n_reads, 96) + 1) / 2 * n_haps;
    return read_bases * 5 + hap_bases * 9 + pairs * (8 + 8 + 1 + sizeof(RerunEntry)) + items * sizeof(WorkItem) +
           n_reads * 11 + n_haps * 9 + 4096;
}

// Validation shared by every entry point: counts, non-decreasing offsets, the reference limits and
// the pointers the batch needs.  Returns PHMM_OK, PHMM_ERR_INVALID_ARGUMENT or
// PHMM_ERR_LIMIT_EXCEEDED (err holds the detail).
phmm_status scan_batch(const phmm_batch& b, const PlanLimits& lim, BatchScan& s, std::string& err);

// scan_batch, then the full plan.  Same return codes.
phmm_status build_plan(const phmm_batch& b, const PlanLimits& lim, Plan& plan, std::string& err);

// Runs covering every pair of a planned batch in the FP64 classes of modes 1 and 2 (whose check kernels take
// any read), of at most max_cols columns where a haplotype is not longer (half of that for multi-stripe
// reads), longest first in a class; cd receives the classes' segments of `all`.  There are no more of them
// than pairs.
void all_pair_runs(const Plan& plan, uint32_t max_cols, std::vector<RerunEntry>& all, std::vector<ClassDesc>& cd);

}  // namespace phmm
