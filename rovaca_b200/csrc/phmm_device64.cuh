// FP64 recompute (the pass that reruns the pairs whose FP32 sum underflowed): the lane state and step
// of the FP32 kernels (phmm_device2.cuh) in scalar double, one read per warp.  LaneRowsEq for constant gap qualities with equal insertion and deletion quality
// (the FP64 classes of mode 0, PM_EQ), LaneRowsRow for per-row gap parameters (modes 1 and 2); the
// all-FP64 check kernels keep phmm_device.cuh's sweep.
//
// Lane state between steps: per row the pending diagonal sum s (M[i][j+1] = s * prior) and
// D[i][j+1]; the lane above forms the lane's first-row I and diagonal sum from its bottom row (mm,
// gapm and mx are one value per read), so a step shuffles two doubles.  Per cell the reference's
// operations on the same operands as phmm_device.cuh `cells` (M * mx, formed once, is also M * my
// since mx == my), with 2 K + 3 doubles of lane state instead of 4 K + 3, two shuffles instead of three,
// and (PM_EQ) 7 operations per cell instead of 8.  The reference flushes every result below 2^-1022 to 0.
// Here a run is swept without flushes, and its pairs whose sum is below 2^-700 again with a flush after
// every operation: those have the reference's bits by construction, the others as explained at
// kUnflushedMin.
#pragma once

#include "phmm_device.cuh"

namespace phmm {

template <int K>
struct LaneRowsEq {
    double S[K];                    // diagonal sum of row k for the lane's next column
    double Dn[K];                   // D of row k at the lane's next column
    double In, Sn;                  // I of the row below the lane and its diagonal sum (to lane + 1)
    double Mb, Ib;                  // bottom row's M and I (lane 31's sums)
    double xx[K];
    double xxn;                     // xx of the row below the lane (1 for a pad row)
    double mm, gm, mx;              // one value per read (mx == my)
    uint32_t padmask;               // bit k: slot k is a pad row
};

// Loads this lane's rows of the stripe starting at padded row first_padded_row (pad rows above the
// read) and writes their priors to the warp's table.  Returns true when one of the lane's rows is an
// inter row with a byte outside A/C/G/T (see load_rows).
template <int K, int V>
__device__ __forceinline__ bool load_rows_eq(LaneRowsEq<K>& L, double* tab, const BatchView& b,
                                             const ProbTables<double>& tb, uint64_t roff, int R, int first_padded_row,
                                             int pad, int lane)
{
    bool exotic = false;
    L.padmask = 0;
    {
        // constant along the read: its first row gives them (pad rows ignore them)
        const int iq = R > 0 ? b.read_i[roff] & 127 : 0, dq = R > 0 ? b.read_d[roff] & 127 : 0;
        const int c = R > 0 ? b.read_c[roff] & 127 : 0;
        L.mm = tb.mm[iq * 128 + dq];
        L.gm = tb.gapm[c];
        L.mx = tb.ph2pr[iq];
    }
    // for lane 31 the row below is the next stripe's first row
    const int below = first_padded_row + lane * K + K - pad;
    L.xxn = below >= 0 && below < R ? tb.ph2pr[b.read_c[roff + (uint64_t)below] & 127] : 1.0;
    L.In = L.Sn = L.Mb = L.Ib = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        L.S[k] = L.Dn[k] = 0.0;
        const int i = first_padded_row + lane * K + k - pad;  // 0-based read position
        double pa = 0.0, pb = 0.0;  // pad rows: prior 0 for every class
        uint32_t rc = 0u;
        if (i >= 0 && i < R) {
            const uint64_t o = roff + (uint64_t)i;
            const int q = b.read_q[o] & 127;
            pa = tb.pmat[q];
            pb = (V == kInter) ? tb.pmis_inter[q] : tb.pmis_intra[q];
            L.xx[k] = tb.ph2pr[b.read_c[o] & 127];
            const uint8_t base = b.read_bases[o];
            rc = match_code(base, V);
            if (V == kInter) exotic |= base_class(base) == 4u;
        } else {
            L.xx[k] = 1.0;
            L.padmask |= 1u << k;
        }
#pragma unroll
        for (int c = 0; c < kTabClasses; ++c)
            tab[prior_slot<K>((uint32_t)c, k, lane)] = class_matches((uint32_t)c, rc, V) ? pa : pb;
    }
    return exotic;
}

// The same lane state with per-row gap parameters (PM_ROW: the FP64 classes of modes 1 and 2): each
// row's mm, gapm, mx and my, and those of the row below the lane (whose first-row I and diagonal sum
// this lane forms).
template <int K>
struct LaneRowsRow {
    double S[K];
    double Dn[K];
    double In, Sn;
    double Mb, Ib;
    double xx[K], mm[K], gm[K], mx[K], my[K];
    double xxn, mmn, gmn, mxn;      // the row below the lane (xx 1 and the rest 0 for a pad row)
    uint32_t padmask;
};

template <int K, int V>
__device__ __forceinline__ bool load_rows_row(LaneRowsRow<K>& L, double* tab, const BatchView& b,
                                              const ProbTables<double>& tb, uint64_t roff, int R, int first_padded_row,
                                              int pad, int lane)
{
    bool exotic = false;
    L.padmask = 0;
    L.In = L.Sn = L.Mb = L.Ib = 0.0;
    // gap parameters of read row i (a pad row: xx 1, the others 0)
    auto params = [&](int i, double& xx, double& mm, double& gm, double& mx, double& my) {
        if (i >= 0 && i < R) {
            const uint64_t o = roff + (uint64_t)i;
            const int iq = b.read_i[o] & 127, dq = b.read_d[o] & 127, c = b.read_c[o] & 127;
            xx = tb.ph2pr[c];
            mm = tb.mm[iq * 128 + dq];
            gm = tb.gapm[c];
            mx = tb.ph2pr[iq];
            my = tb.ph2pr[dq];
        } else {
            xx = 1.0;
            mm = gm = mx = my = 0.0;
        }
    };
    double myn;
    params(first_padded_row + lane * K + K - pad, L.xxn, L.mmn, L.gmn, L.mxn, myn);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        L.S[k] = L.Dn[k] = 0.0;
        const int i = first_padded_row + lane * K + k - pad;  // 0-based read position
        params(i, L.xx[k], L.mm[k], L.gm[k], L.mx[k], L.my[k]);
        double pa = 0.0, pb = 0.0;  // pad rows: prior 0 for every class
        uint32_t rc = 0u;
        if (i >= 0 && i < R) {
            const uint64_t o = roff + (uint64_t)i;
            const int q = b.read_q[o] & 127;
            pa = tb.pmat[q];
            pb = (V == kInter) ? tb.pmis_inter[q] : tb.pmis_intra[q];
            const uint8_t base = b.read_bases[o];
            rc = match_code(base, V);
            if (V == kInter) exotic |= base_class(base) == 4u;
        } else {
            L.padmask |= 1u << k;
        }
#pragma unroll
        for (int c = 0; c < kTabClasses; ++c)
            tab[prior_slot<K>((uint32_t)c, k, lane)] = class_matches((uint32_t)c, rc, V) ? pa : pb;
    }
    return exotic;
}

template <int V, bool FLUSH>
__device__ __forceinline__ double diag_eq(double gm, double mm, double dgM, double dgI, double dgD)
{
    auto fz = [](double x) { return FLUSH ? ftz(x) : x; };
    if (V == kInter) return fz(rfma(dgD, gm, fz(rfma(dgM, mm, fz(rmul(dgI, gm))))));
    return fz(rfma(dgD, gm, fz(rfma(dgI, gm, fz(rmul(dgM, mm))))));
}

// All K rows of the lane at one column.  upI, upS: the first row's I at this column and its diagonal
// sum for the next column, formed by the lane above; pr: the rows' priors at this column.
template <int K, int V, bool FLUSH>
__device__ __forceinline__ void cells_eq(LaneRowsEq<K>& L, const double (&pr)[K], double upI, double upS)
{
    auto fz = [](double x) { return FLUSH ? ftz(x) : x; };
    double Iab = upI, Pab = 0.0;  // I and M * mx of the row above, this column
    double nM = fz(rmul(L.S[0], pr[0]));
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double M = nM;
        if (k + 1 < K) nM = fz(rmul(L.S[k + 1], pr[k + 1]));  // before S[k + 1] is overwritten below
        const double I = k == 0 ? upI : fz(rfma(Iab, L.xx[k], Pab));
        const double D = L.Dn[k];
        Pab = fz(rmul(M, L.mx));
        L.Dn[k] = fz(rfma(D, L.xx[k], Pab));
        const double s = diag_eq<V, FLUSH>(L.gm, L.mm, M, I, D);
        if (k + 1 < K) {
            L.S[k + 1] = s;
        } else {
            L.Mb = M;
            L.Ib = I;
            L.Sn = s;
            L.In = fz(rfma(I, L.xxn, Pab));
        }
        Iab = I;
    }
    L.S[0] = upS;
}

// The same step with per-row gap parameters (8 operations per cell: M * mx of the row below and
// M * my of the row differ).
template <int K, int V, bool FLUSH>
__device__ __forceinline__ void cells_eq(LaneRowsRow<K>& L, const double (&pr)[K], double upI, double upS)
{
    auto fz = [](double x) { return FLUSH ? ftz(x) : x; };
    double Mab = 0.0, Iab = upI;  // the row above, this column
    double nM = fz(rmul(L.S[0], pr[0]));
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double M = nM;
        if (k + 1 < K) nM = fz(rmul(L.S[k + 1], pr[k + 1]));
        const double I = k == 0 ? upI : fz(rfma(Iab, L.xx[k], fz(rmul(Mab, L.mx[k]))));
        const double D = L.Dn[k];
        L.Dn[k] = fz(rfma(D, L.xx[k], fz(rmul(M, L.my[k]))));
        if (k + 1 < K) {
            L.S[k + 1] = diag_eq<V, FLUSH>(L.gm[k + 1], L.mm[k + 1], M, I, D);
        } else {
            L.Mb = M;
            L.Ib = I;
            L.Sn = diag_eq<V, FLUSH>(L.gmn, L.mmn, M, I, D);
            L.In = fz(rfma(I, L.xxn, fz(rmul(M, L.mxn))));
        }
        Mab = M;
        Iab = I;
    }
    L.S[0] = upS;
}

// A row's diagonal sum from (M, I, D) of the row above (flushed), with that row's gap parameters.
template <int V, int K>
__device__ __forceinline__ double row_diag(const LaneRowsEq<K>& L, int, double dgM, double dgI, double dgD)
{
    return diag_eq<V, true>(L.gm, L.mm, dgM, dgI, dgD);
}
template <int V, int K>
__device__ __forceinline__ double row_diag(const LaneRowsRow<K>& L, int k, double dgM, double dgI, double dgD)
{
    return diag_eq<V, true>(L.gm[k], L.mm[k], dgM, dgI, dgD);
}

// The pass sweeps without flushes first.  A result below 2^-1022 that the reference flushes to 0 is then
// kept, which can only matter to values near it: every operation adds products with factors of at most 1,
// so what the flushes take away stays below about 2^-1000 in any later value, and a value of 2^-700 or
// more, which has no bits below 2^-753, is the same with and without it, but where a sum of larger values
// lies exactly on a rounding tie, or within 2^-1000 of one: then its last bit may differ from the
// reference's (one in 2^50 operations or fewer; no such pair is known).  A pair whose sum is below 2^-700, a
// likelihood below 1e-517, is swept again with the reference's flush after every operation; so is one whose
// sum is 0.
// Before, every step either flushed (about three integer operations per FP64 operation, more than the
// FP64 work itself) or ran without under a warp vote that no result could fall below 2^-1022, which long
// reads rarely pass: far from a read's alignment there are always values around 2^-1022.  Measured on
// B200, FP64 pass of 24 regions of reads of 257-768 bases 6.2 ms then, 3.0 ms now; of 60 low-quality regions
// 25.1 and 22.6 ms.
#ifndef PHMM_F64_UNFLUSHED_MIN
#define PHMM_F64_UNFLUSHED_MIN 0x1p-700  // (a test builds the CPU emulator with 0: no pair is swept again)
#endif
constexpr double kUnflushedMin = PHMM_F64_UNFLUSHED_MIN;
// What the unflushed sweep leaves as the likelihood of a pair to be swept again (no likelihood is above 0).
__device__ __forceinline__ double sweep_again() { return __longlong_as_double(0x7ff0000000000000ll); }

// Sweep one stripe over the column stream of haplotypes [g_lo, g_hi): as `sweep` (phmm_device.cuh),
// the scratch row holding the handed-on (I, sum) pair per column.  LR: LaneRowsEq or LaneRowsRow.
// MULTI, from_scr, to_scr: as in the FP32 sweep (phmm_device2.cuh), one sweep for first, middle and last
// stripes.  tiny (lane 31): counts the haplotypes whose sum is below kUnflushedMin; without FLUSH they get
// sweep_again() for a likelihood.
template <int K, int V, bool MULTI, bool FLUSH, typename LR>
__device__ void sweep_eq(LR& L, double* tab, const BatchView& b, const ProbTables<double>& tb,
                         const SweepOut& so, uint32_t g_lo, uint32_t g_hi, double* scr, int lane, bool above_row0,
                         bool exotic, uint64_t roff, int R, int row0, bool from_scr, bool to_scr, uint32_t& tiny)
{
    const bool FROM_SCR = MULTI && from_scr, TO_SCR = MULTI && to_scr;
    const uint64_t s0 = b.hap_off[g_lo];
    const int Tcols = (int)(b.hap_off[g_hi] - s0);
    const uint32_t* codes = (V == kInter ? b.codes_inter : b.codes_intra) + kCodePad + s0;
    const double C = Scale<double>::initial();

    uint32_t cur = g_lo;
    int nb = 0;
    bool started = false;
    double D0 = 0.0;
    double Stop = 0.0;  // lane 0's first-row sum below the boundary row (M = I = 0, D = C/H)
    double sumM = 0.0, sumI = 0.0;
    uint32_t wn = codes[-lane];  // the code word of the lane's next column, loaded a step ahead

    const int steps = Tcols + kWarp;
    // Stripes after the first: the row above (scratch, one 16-byte pair per column) comes through a ring
    // in shared memory, copied two blocks ahead, so that lane 0 does not wait for L2 in every step.
    // Lane 31 writes the same row 31 columns behind lane 0 (for the stripe below), never a column still
    // to be read.
    static_assert(!MULTI || K == kMaxK, "the ring is part of the multi-stripe shape's table");
    double* ring = tab + kTabClasses * K * kWarp;
    auto copy_block = [&](int c0) {
        if (lane < kScrBlock64 && c0 + lane < Tcols) {
            const int c = c0 + lane;
            copy_16_async(&ring[2 * (c & (kScrRing64 - 1))], scr + 2 * c);
        }
        copies_commit();
    };
    if (FROM_SCR) {
        copy_block(0);
        copy_block(kScrBlock64);
    }

    auto boundary = [&]() {
        if (started) {
            if (!TO_SCR && lane == kWarp - 1) {
                // (sums of flushed non-negative values are 0 or normal: no flush needed)
                const double tot = radd(sumM, sumI);
                const uint64_t oi = so.out_base + (uint64_t)(cur - g_lo) * so.out_stride;
                const bool small = !(tot >= kUnflushedMin);
                so.out[oi] = !FLUSH && small ? sweep_again() : log10(tot) - Scale<double>::log10_initial();
                tiny += small;
            }
            ++cur;
        }
        started = true;
        if (cur < g_hi) {
            const int H = (int)(b.hap_off[cur + 1] - b.hap_off[cur]);
            nb += H;
            D0 = C / (double)H;
            // Left edge of the new haplotype: column 0 has M = I = 0 in every row, D = 0 in real rows
            // and C/H in pad rows (which stand for the boundary row, as does the row above the lane's
            // first row when above_row0).  The first column starts from the diagonal sums of column 0
            // and from D[i][1] = fma(D[i][0], xx, 0 * my): C/H in pad rows (xx = 1), else 0.
            Stop = row_diag<V, K>(L, 0, 0.0, 0.0, D0);
            double Dab = above_row0 ? D0 : 0.0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const double Dc = ((L.padmask >> k) & 1u) ? D0 : 0.0;
                L.S[k] = row_diag<V, K>(L, k, 0.0, 0.0, Dab);
                L.Dn[k] = Dc;
                Dab = Dc;
            }
            sumM = 0.0;
            sumI = 0.0;
        } else {
            nb = 0x7fffffff;
        }
    };

    auto step = [&](int t, bool check) {
        const int p = t - lane;
        double uI = shfl_up1(L.In);
        double uS = shfl_up1(L.Sn);
        if (check && p == nb) boundary();
        if (lane == 0) {
            // below the boundary row: I = fma(0, xx, 0 * mx) = 0
            uI = 0.0;
            uS = Stop;
            if (FROM_SCR) {
                const bool ok = p >= 0 && p < Tcols;
                uI = ok ? ring[2 * (p & (kScrRing64 - 1)) + 0] : 0.0;
                uS = ok ? ring[2 * (p & (kScrRing64 - 1)) + 1] : 0.0;
            }
        }
        const uint32_t w = wn;
        wn = codes[p + 1];
        const uint32_t cls = (w & kTabMask) >> kTabShift;
        double pr[K];
#pragma unroll
        for (int k = 0; k < K; ++k) pr[k] = tab[prior_slot<K>(cls, k, lane)];
        if (V == kInter && exotic && cls == 4u) {
            const uint32_t hb = w & kCodeMatchMask;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int i = row0 + lane * K + k;
                if (i >= 0 && i < R && b.read_bases[roff + i] == hb) pr[k] = tb.pmat[b.read_q[roff + i] & 127];
            }
        }
        cells_eq<K, V, FLUSH>(L, pr, uI, uS);
        if (TO_SCR) {
            if (lane == kWarp - 1 && p >= 0 && p < Tcols) {
                scr[2 * p + 0] = L.In;
                scr[2 * p + 1] = L.Sn;
            }
        }
        sumM = radd(sumM, L.Mb);  // (of the last stripe)
        sumI = radd(sumI, L.Ib);
    };
    static_assert(kScrBlock64 % kChunkScalar == 0, "a block of the ring is whole chunks");

    // A flushed step is four times the instructions of an unflushed one (three integer operations behind
    // every FP64 operation), and its loop is kept rolled: unrolled by four as the other the
    // call took 61.5 instead of 54.8 ms (B200, 96,000 pairs below 2^-700, each swept both ways).
    for (int t0 = 0; t0 < steps; t0 += kChunkScalar) {
        if (FROM_SCR && t0 % kScrBlock64 == 0) {  // columns up to t0 + 2 blocks are complete from here
            copies_wait_all();
            __syncwarp();
            copy_block(t0 + 2 * kScrBlock64);
        }
        const int nb31 = __shfl_sync(0xffffffffu, nb, kWarp - 1);
        if (nb31 >= t0 + kChunkScalar && t0 + kChunkScalar <= steps) {
#pragma unroll(FLUSH ? 1 : kChunkScalar)
            for (int u = 0; u < kChunkScalar; ++u) step(t0 + u, false);
        } else {
#pragma unroll 1
            for (int u = 0; u < kChunkScalar; ++u)
                if (t0 + u < steps) step(t0 + u, true);
        }
    }
    if (FROM_SCR) {
        copies_wait_all();
        __syncwarp();
    }
}

}  // namespace phmm
