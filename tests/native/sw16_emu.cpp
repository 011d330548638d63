// The two-alignments-per-warp Smith-Waterman device code (rovaca_b200/csrc/phmm_sw16.cuh) compiled by g++
// and run on 32 host threads standing for the lanes: shuffles and votes go through a per-warp slot
// array and a barrier, shared memory and scratch are heap blocks with guard bytes that are checked.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

namespace {
struct Warp {
    std::atomic<int> count{32}, sense{0};
    uint32_t slot[32];
    void meet()
    {
        const int s = sense.load(std::memory_order_relaxed);
        if (count.fetch_sub(1, std::memory_order_acq_rel) == 1) {
            count.store(32, std::memory_order_relaxed);
            sense.store(s ^ 1, std::memory_order_release);
        } else {
            while (sense.load(std::memory_order_acquire) == s) std::this_thread::yield();
        }
    }
};
thread_local Warp* t_warp;
thread_local int t_lane;
uint32_t give(uint32_t v, int src)
{
    t_warp->slot[t_lane] = v;
    t_warp->meet();
    const uint32_t r = t_warp->slot[src];
    t_warp->meet();
    return r;
}
uint32_t __shfl_up_sync(unsigned, uint32_t v, int d) { return give(v, t_lane >= d ? t_lane - d : t_lane); }
uint32_t __shfl_sync(unsigned, uint32_t v, int src) { return give(v, src); }
uint32_t __shfl_xor_sync(unsigned, uint32_t v, int m) { return give(v, t_lane ^ m); }
uint32_t __ballot_sync(unsigned, bool p)
{
    t_warp->slot[t_lane] = p;
    t_warp->meet();
    uint32_t m = 0;
    for (int k = 0; k < 32; ++k) m |= t_warp->slot[k] << k;
    t_warp->meet();
    return m;
}
bool __any_sync(unsigned, bool p) { return __ballot_sync(0, p) != 0; }
void __syncwarp() { t_warp->meet(); }
int __ffs(int x) { return __builtin_ffs(x); }
}  // namespace

#include "../../rovaca_b200/csrc/phmm_sw16.cuh"

using namespace phmm;

namespace {
constexpr size_t kGuard = 512;
struct Block {  // a zeroed, 256-byte aligned block with guard bytes on both sides
    std::vector<char> mem;
    char* p;
    size_t n;
    explicit Block(size_t bytes) : mem(bytes + 2 * kGuard + 256, 0x5a), n(bytes)
    {
        p = (char*)(((uintptr_t)mem.data() + kGuard + 255) & ~(uintptr_t)255);
        std::memset(p, 0, n);
    }
    bool intact() const
    {
        for (const char* q = mem.data(); q < mem.data() + mem.size(); ++q)
            if ((q < p || q >= p + n) && *q != 0x5a) return false;
        return true;
    }
};

template <int K, bool REB>
bool run(SwView v, uint32_t ix, uint32_t iy, uint32_t max_rows)
{
    Block scr(sw16_layout(max_rows, K).total), sm(Sw16Shared<K, REB>::bytes(max_rows));
    Warp w;
    std::vector<std::thread> lanes;
    for (int l = 0; l < 32; ++l)
        lanes.emplace_back([&, l] {
            t_warp = &w;
            t_lane = l;
            sw16_pair<K, REB>(v, ix, iy, l, (uint8_t*)scr.p, sm.p, max_rows);
        });
    for (auto& t : lanes) t.join();
    return scr.intact() && sm.intact();
}
}  // namespace

// The form (SwForm) width K runs these alignments in.
extern "C" int emu_sw16_form(const int32_t* prm, int i32, uint32_t nrow, uint32_t ncol, int K)
{
    return sw_form(SwParams{prm[0], prm[1], prm[2], prm[3]}, i32 != 0, nrow, ncol, K);
}

// Runs items (0, 1), or item 0 alone (n == 1), in the plain or the rebased form; results and up to `cap` CIGAR ops per item.  0 when the
// code stayed inside its buffers.
extern "C" int emu_sw16(int K, int rebased, const int32_t* prm, int variant, int n, const SwItem* items, const uint8_t* hap,
                        const uint8_t* read, uint32_t cap, phmm_sw_result* out, uint32_t* ops)
{
    SwView v{};
    v.items = items;
    v.hap = hap;
    v.read = read;
    v.prm = SwParams{prm[0], prm[1], prm[2], prm[3]};
    v.variant = variant;
    v.out = out;
    const uint64_t slots[2] = {0, cap};
    v.slot_off = slots;
    v.ops = ops;
    v.cigar_cap = cap;
    uint32_t rows = 0;
    for (int q = 0; q < n; ++q) rows = rows > items[q].hap_len ? rows : items[q].hap_len;
    const uint32_t iy = n > 1 ? 1u : 0xffffffffu;
    switch (K) {
    case 1: return rebased ? !run<1, true>(v, 0, iy, rows) : !run<1, false>(v, 0, iy, rows);
    case 3: return rebased ? !run<3, true>(v, 0, iy, rows) : !run<3, false>(v, 0, iy, rows);
    case 5: return rebased ? !run<5, true>(v, 0, iy, rows) : !run<5, false>(v, 0, iy, rows);
    case 8: return rebased ? !run<8, true>(v, 0, iy, rows) : !run<8, false>(v, 0, iy, rows);
    case 10: return rebased ? !run<10, true>(v, 0, iy, rows) : !run<10, false>(v, 0, iy, rows);
    case 24: return rebased ? !run<24, true>(v, 0, iy, rows) : !run<24, false>(v, 0, iy, rows);
    default: return 2;
    }
}
