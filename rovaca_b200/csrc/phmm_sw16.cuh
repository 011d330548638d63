// Smith-Waterman of two alignments per warp in 16-bit halves.  The recurrences, tie rules, end-cell
// choice and trace-back are those of phmm_sw.cu (reference: common/base/lib/ro_sw/sw_core_template.h:
// 111-352, sw_cigar.c:22-171); this is the form for alignments whose scores, or whose scores' differences
// within a lane, fit 16 bits whatever the bases (sw_form: the genotyping and the assembly parameters up to
// 768 read bases), so that no add can wrap and the reference's int16 and int32 kernels give the same
// results.
//
// Mapping.  Alignment X in the low and Y in the high half of every 32-bit register.  Lane l holds K
// read columns of both and works on row t + 1 - l at step t; the left neighbour's H and E arrive by one
// shuffle each.  The columns are padded at the front to 32 * K, so that the last read column of both
// sits in lane 31's last slot: a pad column scores 0 against every base, which with gap_open <= 0 and
// gap_extend < 0 keeps H = 0 and E = gap_open in it, the values the boundary column stands for.
//
// Arithmetic.  Scores are stored with a bias that makes every half non-negative, so that a packed add
// or subtract is one plain 32-bit instruction (no borrow crosses the halves) and only the maxima are
// packed instructions.  The four facts of a cell (E extended, F extended, H equals the diagonal term, H
// equals E; a tie goes to the diagonal, then to the insertion, as the reference's strict comparisons have
// it) come out as sign bits of 0x8000 + a - max; a byte permute that replicates the signs collects two of
// them for both alignments, one AND-OR deposits them: 4 operations per packed cell for the codes, 15 in
// all, 7.5 per cell against about 21 in the 32-bit kernel.
// The substitution scores come from a per-lane table in shared memory (6 base classes x K columns per
// alignment: A, C, G, T, N, any other byte) read at the row's class, one permute per packed cell to
// join the halves; a read with a byte outside A/C/G/T/N runs the comparing form of the step.
// Bound: integer ALU issue (75% of the pipe's cycles at 16 warps per SM; long-scoreboard and
// shared-memory waits below half a cycle per issue).  Measured on B200 on 74,776 alignments (300 regions
// of the benchmark's shape, 4.91e9 cells), device time alone: 8.53 ms with one alignment per warp in 32
// bits, 2.97 ms here (1,650 GCUPS).
//
// Trace-back.  Lanes 0-15 follow X and lanes 16-31 Y.  Each iteration the 16 lanes look at the next 16
// cells in the direction of the state (diagonal, or along the gap) and take the whole run at once.
#pragma once

#include <cstdint>

#include "phmm_sw.h"

namespace phmm {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t sw_max3(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_u16x2(a, b, c); }
// max(a + b, c) per half (the add wraps per half: b may be a negated constant)
__device__ __forceinline__ uint32_t sw_addmax2(uint32_t a, uint32_t b, uint32_t c) { return __viaddmax_u16x2(a, b, c); }
template <uint32_t SEL>
__device__ __forceinline__ uint32_t sw_prmt(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "n"(SEL));
    return d;
}
#else
__device__ inline uint32_t sw_max2(uint32_t a, uint32_t b)
{
    const uint32_t l = (a & 0xffffu) > (b & 0xffffu) ? a & 0xffffu : b & 0xffffu;
    const uint32_t h = (a >> 16) > (b >> 16) ? a >> 16 : b >> 16;
    return l | (h << 16);
}
__device__ inline uint32_t sw_max3(uint32_t a, uint32_t b, uint32_t c) { return sw_max2(sw_max2(a, b), c); }
__device__ inline uint32_t sw_addmax2(uint32_t a, uint32_t b, uint32_t c)
{
    return sw_max2(((a + b) & 0xffffu) | ((a & 0xffff0000u) + (b & 0xffff0000u)), c);
}
template <uint32_t SEL>
__device__ inline uint32_t sw_prmt(uint32_t a, uint32_t b)
{
    uint32_t r = 0;
    for (int k = 0; k < 4; ++k) {
        const uint32_t s = (SEL >> (4 * k)) & 15u, src = s & 7u;
        uint32_t byte = (src < 4 ? a >> (8 * src) : b >> (8 * (src - 4))) & 0xffu;
        if (s & 8u) byte = byte & 0x80u ? 0xffu : 0u;
        r |= byte << (8 * k);
    }
    return r;
}
#endif

struct Sw16True {
    static constexpr bool value = true;
};
struct Sw16False {
    static constexpr bool value = false;
};

constexpr int kSw16Planes = 6;  // A, C, G, T, N, any other byte

PHMM_HD inline uint32_t sw16_class(uint8_t b)
{
    return b == 'A' ? 0u : b == 'C' ? 1u : b == 'G' ? 2u : b == 'T' ? 3u : b == 'N' ? 4u : 5u;
}

// Steps between two rebasings of the rebased form (see sw16_pair).
constexpr int kSw16Rebase = 32;

// Shared memory of one warp: the two score tables (per class and 16-byte group of 8 columns, one uint4
// per lane), the last row (per padded column) and last column (per row), packed, or one i32 each for X
// and Y in the rebased form, and the rows' base classes (one u16 per row, X in the low byte, 32 spare
// rows on both sides).
template <int K, bool REB>
struct Sw16Shared {
    static constexpr int NV = (K + 7) / 8;
    static constexpr int kWords = REB ? 2 : 1;                    // per row and per column
    static constexpr uint32_t kPlane = NV * 512;                  // bytes
    static constexpr uint32_t kTable = kSw16Planes * kPlane;      // bytes, per alignment
    static constexpr uint32_t lrow_off = 2 * kTable;
    static constexpr uint32_t lcol_off = lrow_off + 32 * K * 4 * kWords;
    PHMM_HD static uint32_t rows_off(uint32_t max_rows) { return lcol_off + ((max_rows + 4) & ~3u) * 4 * kWords; }
    PHMM_HD static uint32_t bytes(uint32_t max_rows) { return (rows_off(max_rows) + (max_rows + 64) * 2 + 15) & ~15u; }
};

struct Sw16Half {
    const uint8_t* hap;
    const uint8_t* read;
    int nrow, ncol, pad;
    uint32_t idx;
    bool live;      // has rows and columns (an empty sequence is settled without the sweep)
    bool write;     // false: stands in for a missing second alignment
    bool i32;
};

// The end cell among the cells of the last row (row(j), j = 1..ncol) and column (col(i), i = 1..nrow)
// that reach the maximum, visited in the reference's order (anti-diagonal ascending; the last-row cell
// before the last-column cell).
template <typename Row, typename Col>
__device__ inline void sw16_end_cell(int nrow, int ncol, Row row, Col col, int lane, int& best, int& mi, int& mj)
{
    int smax = (int)0x80000000;
    for (int j = 1 + lane; j <= ncol; j += 32) smax = row(j) > smax ? row(j) : smax;
    for (int i = 1 + lane; i <= nrow; i += 32) smax = col(i) > smax ? col(i) : smax;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int x = (int)__shfl_xor_sync(0xffffffffu, (uint32_t)smax, o);
        smax = x > smax ? x : smax;
    }
    const int alo = (nrow < ncol ? nrow : ncol) + 1, ahi = nrow + ncol;
    for (int a0 = alo; a0 <= ahi; a0 += 32) {
        const int a = a0 + lane;
        const bool rc = a <= ahi && a >= nrow + 1 && row(a - nrow) == smax;
        const bool cc = a <= ahi && a >= ncol + 1 && col(a - ncol) == smax;
        uint32_t mr = __ballot_sync(0xffffffffu, rc), mc = __ballot_sync(0xffffffffu, cc);
        while (mr | mc) {
            const int l = __ffs((int)(mr | mc)) - 1;
            const int aa = a0 + l;
            if ((mr >> l) & 1u) {
                const int ci = nrow, cj = aa - nrow;
                if (best < smax || abs(ci - cj) < abs(mi - mj)) { best = smax; mi = ci; mj = cj; }
            }
            if ((mc >> l) & 1u) {
                const int ci = aa - ncol, cj = ncol;
                if (best < smax || mj == ncol || abs(ci - cj) <= abs(mi - mj)) { best = smax; mi = ci; mj = cj; }
            }
            mr &= ~(1u << l);
            mc &= ~(1u << l);
        }
    }
}

__device__ inline uint32_t sw16_op(uint32_t run)
{
    const uint32_t st = run >> 16, len = run & 0xffffu;  // state 0 M, 1 I, 2 D, 9 S
    return (len << 4) | (st == 0 ? 0u : st == 1 ? 1u : st == 2 ? 2u : 4u);
}

// Two alignments of one class (K read columns per lane).  scr: the warp's scratch, sm: its shared
// memory; max_rows: the launch's longest haplotype (sizes both).
//
// REB: the rebased form, for scores beyond 16 bits (the assembly parameters).  Neighbouring H differ by
// at most match - gap_open (down to gap_open), so what a lane holds lies within K + 1 such steps of its
// first column, and moves by one more per row.  Each lane keeps a 32-bit base per alignment and the
// halves hold the difference to it plus 32768; every kSw16Rebase steps all lanes move their base to their
// first column's H.  A shuffled value is brought to the receiver's base by one add (the bases' difference,
// exchanged at the rebasing).  Last row and column are kept as 32-bit scores.  Measured on B200, device
// time of 2,726 haplotype-to-window alignments with the assembly parameters: 4.48 ms with one alignment
// per warp in 32 bits (codes by haplotype row), 0.88 ms here.
template <int K, bool REB>
__device__ inline void sw16_pair(const SwView& v, uint32_t ix, uint32_t iy, int lane, uint8_t* scr, char* sm,
                                 uint32_t max_rows)
{
    using SM = Sw16Shared<K, REB>;
    constexpr int NV = SM::NV, NW = (K + 3) / 4, ROW = 32 * NW, S = 32 * K;
    constexpr uint32_t kSign = 0x80008000u;
    const int open = v.prm.gap_open, ext = v.prm.gap_extend, mis = v.prm.mismatch;
    const int bias = REB ? 32768 : sw16_bias(v.prm, K);
    const uint32_t H0 = (uint32_t)bias * 0x10001u;
    const uint32_t LOW = (uint32_t)(bias + open - ext - 1) * 0x10001u;     // extending it stays below opening
    const uint32_t XE = (uint32_t)(-ext) * 0x10001u;
    const uint32_t NO = (uint32_t)(uint16_t)(short)open * 0x10001u;        // + open per half
    const uint32_t MM = (uint32_t)((long long)mis * 0x10001ll);            // + mismatch, linear in the halves

    Sw16Half hf[2];
    int R = 0, Rmin = 0x7fffffff;
    bool exotic = false;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        Sw16Half& h = hf[q];
        h.write = q == 0 || iy != 0xffffffffu;
        h.idx = q == 0 || iy == 0xffffffffu ? ix : iy;
        const SwItem it = v.items[h.idx];
        h.nrow = (int)it.hap_len;
        h.ncol = (int)it.read_len;
        h.i32 = sw_uses_int32(v.variant, it.hap_len, it.read_len, v.prm.match);
        h.live = h.nrow > 0 && h.ncol > 0;
        h.hap = v.hap + it.hap_start;
        h.read = v.read + it.read_start;
        h.pad = S - h.ncol;
        if (h.live) {
            R = R > h.nrow ? R : h.nrow;
            Rmin = Rmin < h.nrow ? Rmin : h.nrow;
        }
    }
    if (!(hf[0].live && hf[1].live)) Rmin = 0;
    uint32_t* lrow = (uint32_t*)(sm + SM::lrow_off);
    uint32_t* lcol = (uint32_t*)(sm + SM::lcol_off);
    uint16_t* rows = (uint16_t*)(sm + SM::rows_off(max_rows));
    uint32_t* bt = (uint32_t*)scr;

    if (R > 0) {
        // score tables (s - mismatch: 0, match - mismatch, or -mismatch in a pad column) and row classes
        const uint32_t hit = (uint32_t)(v.prm.match - mis), padv = (uint32_t)(-mis);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const Sw16Half& h = hf[q];
            uint16_t* tab = (uint16_t*)(sm + q * SM::kTable);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int j = lane * K + k - h.pad;  // 0-based read position
                const bool real = h.live && j >= 0;
                const uint32_t c = real ? sw16_class(h.read[j]) : 0u;
                if (real && c == 5u) exotic = true;
#pragma unroll
                for (int p = 0; p < kSw16Planes; ++p)
                    tab[((p * NV + k / 8) * 32 + lane) * 8 + k % 8] = (uint16_t)(!real ? padv : (int)c == p && p < 5 ? hit : 0u);
            }
        }
        exotic = __any_sync(0xffffffffu, exotic);
        for (int i = lane - 32; i < R + 32; i += 32) {
            uint32_t c[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const bool in = hf[q].live && i >= 0 && i < hf[q].nrow;
                const uint8_t b = in ? hf[q].hap[i] : 0;
                c[q] = exotic ? b : in ? sw16_class(b) : 5u;
            }
            rows[i + 32] = (uint16_t)(c[0] | (c[1] << 8));
        }
        __syncwarp();

        uint32_t Hp[K], Fp[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            Hp[k] = H0;
            Fp[k] = LOW;
        }
        uint32_t hprev = H0, hout = H0, eout = LOW;
        int base_x = 0, base_y = 0;              // REB: this lane's bases
        uint32_t to_mine = 0, edge = 0;          // REB: from the left lane's base (lane 0: from 0) to mine
        auto rebase = [&] {
            const int dx = (int)(Hp[0] & 0xffffu) - 32768, dy = (int)(Hp[0] >> 16) - 32768;
            const uint32_t d = (uint32_t)dx + ((uint32_t)dy << 16);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                Hp[k] -= d;
                Fp[k] -= d;
            }
            hprev -= d;
            hout -= d;
            eout -= d;
            base_x += dx;
            base_y += dy;
            const uint32_t px = __shfl_up_sync(0xffffffffu, (uint32_t)base_x, 1);
            const uint32_t py = __shfl_up_sync(0xffffffffu, (uint32_t)base_y, 1);
            to_mine = (px - (uint32_t)base_x) + ((py - (uint32_t)base_y) << 16);
            edge = 0u - (uint32_t)base_x - ((uint32_t)base_y << 16);
        };
        const char* tx = sm + lane * 16;
        const char* ty = tx + SM::kTable;
        const int capX = hf[0].live ? hf[0].nrow : -1, capY = hf[1].live ? hf[1].nrow : -1;
        // one wavefront step; FULL: every lane is on a row of both alignments before the last one
        auto step = [&](int t, auto full, auto raw) {
            constexpr bool FULL = decltype(full)::value, RAW = decltype(raw)::value;
            const int i = t + 1 - lane;
            if (REB && t % kSw16Rebase == 0 && t > 0) rebase();
            uint32_t hl = __shfl_up_sync(0xffffffffu, hout, 1) + to_mine;
            uint32_t el = __shfl_up_sync(0xffffffffu, eout, 1) + to_mine;
            if (lane == 0) {
                hl = H0 + edge;
                el = LOW + edge;
            }
            const uint32_t cw = rows[t - lane + 32];
            uint32_t wx[4 * NV], wy[4 * NV];
            if (!RAW) {
                const char* px = tx + (cw & 0xffu) * SM::kPlane;
                const char* py = ty + (cw >> 8) * SM::kPlane;
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    const uint4 a = *(const uint4*)(px + q * 512), b = *(const uint4*)(py + q * 512);
                    wx[4 * q] = a.x;
                    wx[4 * q + 1] = a.y;
                    wx[4 * q + 2] = a.z;
                    wx[4 * q + 3] = a.w;
                    wy[4 * q] = b.x;
                    wy[4 * q + 1] = b.y;
                    wy[4 * q + 2] = b.z;
                    wy[4 * q + 3] = b.w;
                }
            }
            const bool act = FULL || i >= 1;
            uint32_t diag = hprev;
            hprev = hl;
            uint32_t code[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) code[w] = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                uint32_t sc;
                if (RAW) {
                    uint32_t s2[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int j = lane * K + k - hf[q].pad;
                        const uint32_t hb = q ? cw >> 8 : cw & 0xffu;
                        s2[q] = !hf[q].live || j < 0 ? (uint32_t)(-mis)
                                                     : (hb == hf[q].read[j] ? (uint32_t)(v.prm.match - mis) : 0u);
                    }
                    sc = s2[0] | (s2[1] << 16);
                } else {
                    sc = k & 1 ? sw_prmt<0x7632>(wx[k / 2], wy[k / 2]) : sw_prmt<0x5410>(wx[k / 2], wy[k / 2]);
                }
                const uint32_t ee = el - XE;
                const uint32_t e = sw_addmax2(hl, NO, ee);
                const uint32_t fe = Fp[k] - XE;
                const uint32_t f = sw_addmax2(Hp[k], NO, fe);
                const uint32_t hr = diag + sc + MM;
                const uint32_t h2 = sw_max3(hr, e, f);
                const uint32_t w1 = sw_prmt<0xFDB9>(kSign + ee - e, kSign + fe - f);    // extended: E, F
                const uint32_t w2 = sw_prmt<0xFDB9>(kSign + hr - h2, kSign + e - h2);   // H is the diagonal, is E
                code[k / 4] |= w1 & (0x01010101u << (2 * (k & 3)));
                code[k / 4] |= w2 & (0x02020202u << (2 * (k & 3)));
                diag = Hp[k];
                if (act) {
                    Hp[k] = h2;
                    Fp[k] = f;
                }
                hl = h2;
                el = e;
            }
            hout = act ? hl : H0;  // a lane before its first row stands for row 0
            eout = act ? el : LOW;
            if (FULL || (i >= 1 && i <= R)) {
                uint32_t* row = bt + (uint32_t)t * ROW + lane;
#pragma unroll
                for (int w = 0; w < NW; ++w) row[w * 32] = code[w];
                if (lane == 31) {
                    if (REB) {
                        lcol[2 * i] = (hl & 0xffffu) - 32768u + (uint32_t)base_x;
                        lcol[2 * i + 1] = (hl >> 16) - 32768u + (uint32_t)base_y;
                    } else {
                        lcol[i] = hl;
                    }
                }
                if (!FULL && REB) {
                    if (i == capX) {
#pragma unroll
                        for (int k = 0; k < K; ++k) lrow[2 * (lane * K + k)] = (Hp[k] & 0xffffu) - 32768u + (uint32_t)base_x;
                    }
                    if (i == capY) {
#pragma unroll
                        for (int k = 0; k < K; ++k) lrow[2 * (lane * K + k) + 1] = (Hp[k] >> 16) - 32768u + (uint32_t)base_y;
                    }
                } else if (!FULL) {
                    if (i == capX) {
#pragma unroll
                        for (int k = 0; k < K; ++k) ((uint16_t*)lrow)[2 * (lane * K + k)] = (uint16_t)Hp[k];
                    }
                    if (i == capY) {
#pragma unroll
                        for (int k = 0; k < K; ++k) ((uint16_t*)lrow)[2 * (lane * K + k) + 1] = (uint16_t)(Hp[k] >> 16);
                    }
                }
            }
        };
        const int steps = R + 31;
        const auto yes = Sw16True{};
        const auto no = Sw16False{};
        int t = 0;
        if (!exotic) {
            const int full_end = Rmin - 1;  // lane 0 reaches row Rmin at step Rmin - 1
            for (; t < steps && t < 31; ++t) step(t, no, no);
            for (; t < full_end; ++t) step(t, yes, no);
            for (; t < steps; ++t) step(t, no, no);
        } else {
            for (; t < steps; ++t) step(t, no, yes);
        }
        __syncwarp();
    }

    int bestv[2], mi[2] = {0, 0}, mj[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const Sw16Half& h = hf[q];
        bestv[q] = h.i32 ? (int)0x80000000 : -32768;
        if (h.live) {
            // row j is padded column pad + j - 1
            auto row = [&](int j) {
                const int c = h.pad + j - 1;
                return REB ? (int)lrow[2 * c + q] : (int)((lrow[c] >> (16 * q)) & 0xffffu) - bias;
            };
            auto col = [&](int i) { return REB ? (int)lcol[2 * i + q] : (int)((lcol[i] >> (16 * q)) & 0xffffu) - bias; };
            sw16_end_cell(h.nrow, h.ncol, row, col, lane, bestv[q], mi[q], mj[q]);
        } else {  // only boundary cells (H = 0), or no candidate at all
            if (h.nrow == 0 && h.ncol > 0) { bestv[q] = 0; mj[q] = 1; }
            if (h.ncol == 0 && h.nrow > 0) { bestv[q] = 0; mi[q] = h.nrow; }
        }
    }

    // trace-back (sw_cigar.c:36-146): half-warp q follows alignment q; runs merged as they come
    const int q = lane >> 4, l16 = lane & 15, base = q * 16;
    const int ncol = q ? hf[1].ncol : hf[0].ncol, pad = q ? hf[1].pad : hf[0].pad;
    const bool write = q ? hf[1].write : hf[0].write;
    const uint32_t idx = q ? hf[1].idx : hf[0].idx;
    const Sw16Layout L = sw16_layout(max_rows, K);
    uint32_t* runs = (uint32_t*)(scr + L.runs + (uint64_t)q * L.run_stride);
    int i = q ? mi[1] : mi[0], j = q ? mj[1] : mj[0];
    const int end_i = i, end_j = j, best = q ? bestv[1] : bestv[0];
    int nr = 0, cst = -1, clen = 0;
    auto push = [&](int st, int len) {
        if (nr > 0 && cst == st) {
            clen += len;
        } else {
            if (nr > 0 && l16 == 0) runs[nr - 1] = ((uint32_t)cst << 16) | (uint32_t)clen;
            cst = st;
            clen = len;
            ++nr;
        }
    };
    if (j < ncol) push(9, ncol - j);
    int state = 0;  // 0 on the diagonal, 1 inside an insertion (along the row), 2 inside a deletion
    while (__any_sync(0xffffffffu, i > 0 && j > 0)) {
        const int ci = i - (state == 1 ? 0 : l16), cj = j - (state == 2 ? 0 : l16);
        const bool in = ci > 0 && cj > 0 && i > 0 && j > 0;
        uint32_t b = 0;  // bit 0 E extended, 1 H is the diagonal term, 2 F extended, 3 H is E
        if (in) {
            const int s = cj - 1 + pad, ln = s / K, k = s - ln * K;
            const uint32_t w = bt[(uint32_t)(ci - 1 + ln) * ROW + (k >> 2) * 32 + ln] >> (8 * q + 2 * (k & 3));
            b = (w & 3u) | ((w >> 14) & 12u);
        }
        const bool go = in && (state == 0 ? (b & 2u) != 0 : state == 1 ? (b & 1u) != 0 : (b & 4u) != 0);
        const uint32_t valid = (__ballot_sync(0xffffffffu, in) >> base) & 0xffffu;
        const uint32_t run = (__ballot_sync(0xffffffffu, go) >> base) & 0xffffu;
        const uint32_t b0 = __shfl_sync(0xffffffffu, b, base);
        if (valid) {
            const int cells = __ffs((int)(~valid)) - 1;  // valid lanes are the first ones
            const int n = __ffs((int)(~run)) - 1;
            if (state == 0) {
                if (n > 0) {
                    push(0, n);
                    i -= n;
                    j -= n;
                } else if ((b0 & 8u) == 0) {  // above the diagonal term and E: a deletion
                    push(2, 1);
                    --i;
                    state = b0 & 4u ? 2 : 0;
                } else {
                    push(1, 1);
                    --j;
                    state = b0 & 1u ? 1 : 0;
                }
            } else {
                // the cells that extend, and the one that opened the gap
                const int take = n + 1 < cells ? n + 1 : cells;
                clen += take;
                if (state == 1) j -= take;
                else i -= take;
                if (take > n) state = 0;
            }
        }
    }
    if (j > 0) push(9, j);
    if (nr > 0 && l16 == 0) runs[nr - 1] = ((uint32_t)cst << 16) | (uint32_t)clen;
    __syncwarp();

    // read order, at most kSwMaxSeq - 1 ops (sw_cigar.c:162-170)
    if (write) {
        const int count = nr < kSwMaxSeq - 1 ? nr : kSwMaxSeq - 1;
        const int wr = count < (int)v.cigar_cap ? count : (int)v.cigar_cap;
        uint32_t* dst = v.ops + v.slot_off[idx];
        for (int c = l16; c < wr; c += 16) dst[c] = sw16_op(runs[nr - 1 - c]);
        if (l16 == 0) {
            phmm_sw_result res;
            res.score = best;
            res.alignment_offset = i;
            res.max_i = end_i;
            res.max_j = end_j;
            res.cigar_count = (uint32_t)count;
            res.cigar_offset = 0;
            v.out[idx] = res;
        }
    }
    __syncwarp();
}

}  // namespace phmm
