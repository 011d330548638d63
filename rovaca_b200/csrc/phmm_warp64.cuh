// One warp's share of an FP64 recompute class: the persistent claim loop over the class's runs of
// underflowed pairs, each streamed through its read (phmm_device.cuh).  Device code only: the class
// kernels (phmm_kernels.cu) call it, and it compiles for the host as well, where
// tests/native/warp_emu.cpp runs it on 32 threads standing for the lanes.
#pragma once

#include <type_traits>

#include "phmm_device.cuh"
#include "phmm_device64.cuh"

namespace phmm {

// ------------------------------------------------------------------------------------------
// One read against a run of haplotypes [g_lo, g_hi) in the recompute pass: the two-value lane state
// (phmm_device64.cuh), one value per read for constant gaps with insertion = deletion, per row otherwise.
// FLUSH: with the flush after every operation.  Returns the haplotypes whose sum is below kUnflushedMin.
// ------------------------------------------------------------------------------------------
template <int K, int V, int PM, bool MULTI, bool FLUSH>
__device__ __forceinline__ uint32_t run_stripes(const BatchView& b, const ProbTables<double>& tb, const SweepOut& so,
                                                uint32_t g_lo, uint32_t g_hi, int lane, double* scr, double* tab,
                                                uint64_t roff, int R)
{
    uint32_t tiny = 0;
    using LR = typename std::conditional<PM == PM_EQ, LaneRowsEq<K>, LaneRowsRow<K>>::type;
    LR L;
    constexpr int SR = kWarp * K;  // rows per stripe
    const int stripes = MULTI ? (R + SR - 1) / SR : 1;
    const int pad = SR * stripes - R;
    for (int s = 0; s < stripes; ++s) {
        bool exotic;
        if constexpr (PM == PM_EQ)
            exotic = load_rows_eq<K, V>(L, tab, b, tb, roff, R, s * SR, pad, lane);
        else
            exotic = load_rows_row<K, V>(L, tab, b, tb, roff, R, s * SR, pad, lane);
        const bool above_row0 = (s == 0) && (lane * K <= pad);
        const int row0 = s * SR - pad;  // read position of slot 0 of lane 0
        sweep_eq<K, V, MULTI, FLUSH>(L, tab, b, tb, so, g_lo, g_hi, scr, lane, above_row0, exotic, roff, R, row0, s > 0,
                                     s < stripes - 1, tiny);
        // lane 31's scratch row is read by lane 0 in the next stripe; every lane's priors are rewritten
        __syncwarp();
    }
    return __shfl_sync(0xffffffffu, tiny, kWarp - 1);
}

// The first haplotype from g on (below g_hi, else g_hi) that is, or is not, marked to be swept again.
__device__ __forceinline__ uint32_t next_marked(const SweepOut& so, uint32_t g_lo, uint32_t g, uint32_t g_hi, bool marked,
                                                int lane)
{
    for (; g < g_hi; g += kWarp) {
        const uint32_t h = g + (uint32_t)lane;
        const bool hit = h < g_hi && (so.out[so.out_base + (uint64_t)(h - g_lo) * so.out_stride] == sweep_again()) == marked;
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (m) return g + (uint32_t)__ffs((int)m) - 1u;
    }
    return g_hi;
}

constexpr uint32_t kTinyRuns = 2;

// ------------------------------------------------------------------------------------------
// One read against a run of haplotypes [g_lo, g_hi).
// tiny_runs (recompute pass): the warp's last runs in a row whose pairs were all below kUnflushedMin.  After
// kTinyRuns of them (reads that do not belong to their region come together) the next is swept with the
// flushes at once, which gives the same results and saves the unflushed sweep; where such pairs are few, that
// is hardly ever wrong.  Otherwise only the haplotypes below the line are swept again, each group of
// neighbours by itself.  Measured on B200, one call with every run swept twice, and now: 96,000
// pairs of foreign reads of 250 bases, all below the line, 61.7 and 42.4 ms (1 run: 41.8, 4 runs: 43.4); of
// foreign reads of 600 bases 38.2 and 27.3 ms; 9% of 96,000 pairs below it 25.8 and 24.2 ms (1 run: 25.3).
// ------------------------------------------------------------------------------------------
template <typename T, int K, int V, int PM, bool MULTI, bool UNF = false>
__device__ __forceinline__ void run_read(const BatchView& b, const ProbTables<T>& tb, const PassControl& pc,
                                         const SweepOut& so, uint32_t g_lo, uint32_t g_hi, int lane, T* scr, T* tab,
                                         uint32_t& tiny_runs)
{
    const uint64_t roff = b.read_off[so.read];
    const int R = (int)(b.read_off[so.read + 1] - roff);
    const int Tcols = (int)(b.hap_off[g_hi] - b.hap_off[g_lo]);
    // A read that does not fit the class's stripe, or a multi-stripe stream longer than the
    // scratch row, means a planning bug: report it and leave the pairs as NaN.
    if (R <= 0 || (!MULTI && R > kWarp * K) || (MULTI && (R <= kWarp * K || Tcols > (int)pc.scratch_cols))) {
        if (lane == 0) atomicOr(pc.status, kStatusBadItem);
        return;
    }
    if constexpr (PM == PM_EQ || (PM == PM_ROW && !UNF)) {
        static_assert(sizeof(T) == 8 && !UNF, "the two-value lane state is the FP64 recompute");
        const bool flush_all = tiny_runs >= kTinyRuns;
        uint32_t tiny = 0, lo = g_lo;
        if (!flush_all) {
            tiny = run_stripes<K, V, PM, MULTI, false>(b, tb, so, g_lo, g_hi, lane, scr, tab, roff, R);
            if (tiny == 0) {
                tiny_runs = 0;
                return;
            }
            lo = next_marked(so, g_lo, g_lo, g_hi, true, lane);
        }
        uint32_t flushed_tiny = 0;
        while (lo < g_hi) {
            const uint32_t hi = flush_all ? g_hi : next_marked(so, g_lo, lo, g_hi, false, lane);
            SweepOut part = so;
            part.out_base += (uint64_t)(lo - g_lo) * so.out_stride;
            flushed_tiny += run_stripes<K, V, PM, MULTI, true>(b, tb, part, lo, hi, lane, scr, tab, roff, R);
            lo = flush_all ? g_hi : next_marked(so, g_lo, hi, g_hi, true, lane);
        }
        tiny_runs = (flush_all ? flushed_tiny : tiny) == g_hi - g_lo ? tiny_runs + 1 : 0;
    } else {
        LaneRows<T, K, PM> L;
        if (!MULTI) {
            const int pad = kWarp * K - R;
            const bool exotic = load_rows<T, K, V, PM>(L, tab, b, tb, roff, R, 0, pad, lane);
            sweep<T, K, V, PM, false, false, UNF>(L, tab, b, tb, pc, so, g_lo, g_hi, scr, lane, lane * K <= pad, exotic,
                                                  roff, R, -pad);
        } else {
            constexpr int SR = kWarp * K;  // rows per stripe
            const int stripes = (R + SR - 1) / SR;
            const int pad = SR * stripes - R;
            for (int s = 0; s < stripes; ++s) {
                const bool exotic = load_rows<T, K, V, PM>(L, tab, b, tb, roff, R, s * SR, pad, lane);
                const bool above_row0 = (s == 0) && (lane * K <= pad);
                const int row0 = s * SR - pad;  // read position of slot 0 of lane 0
                if (s == 0)
                    sweep<T, K, V, PM, false, true, UNF>(L, tab, b, tb, pc, so, g_lo, g_hi, scr, lane, above_row0, exotic,
                                                         roff, R, row0);
                else if (s == stripes - 1)
                    sweep<T, K, V, PM, true, false, UNF>(L, tab, b, tb, pc, so, g_lo, g_hi, scr, lane, above_row0, exotic,
                                                         roff, R, row0);
                else
                    sweep<T, K, V, PM, true, true, UNF>(L, tab, b, tb, pc, so, g_lo, g_hi, scr, lane, above_row0, exotic,
                                                        roff, R, row0);
                __syncwarp();  // lane 31's scratch row is read by lane 0 in the next stripe
            }
        }
    }
}

// The claim loop of one warp over the class's rerun segment (pc.cd).  UNF: the all-FP64 check
// arithmetic (plain multiply and add); the recompute pass proper uses the reference's contracted
// arithmetic.  tab: the warp's shared prior table (prior_table_size<K>() values); warp_id: the
// warp's index in the grid (its scratch row).
template <int K, int V, int PM, bool MULTI, bool UNF = false>
__device__ __forceinline__ void warp_reruns64(const BatchView& b, const ProbTables<double>& tb, const PassControl& pc,
                                              double* tab, int lane, unsigned int warp_id)
{
    double* scr = MULTI ? (double*)pc.scratch + (size_t)warp_id * pc.scratch_cols * 3 : nullptr;
    const unsigned int n = min(pc.cd->rerun_count, pc.cd->rerun_cap);
    const RerunEntry* rerun = pc.rerun + pc.cd->rerun_off;
    uint32_t tiny_runs = 0;
    for (;;) {
        const unsigned int idx = claim(&pc.cd->claim64, lane);
        if (idx >= n) break;
        const RerunEntry e = rerun[idx];
        SweepOut so;
        so.out = b.out;
        so.pair_flags = nullptr;
        so.out_base = e.out_idx;
        so.out_stride = e.out_stride;
        so.read = e.read;
        run_read<double, K, V, PM, MULTI, UNF>(b, tb, pc, so, e.hap, e.hap + e.n_haps, lane, scr, tab, tiny_runs);
    }
}

}  // namespace phmm
