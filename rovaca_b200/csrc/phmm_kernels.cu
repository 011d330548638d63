// PairHMM kernels for sm_100a: haplotype code preparation, the persistent FP64 recompute pass, the
// FMA throughput probes and the launch wrappers of every class.  Device arithmetic lives in
// phmm_device.cuh (scalar) and phmm_device2.cuh (packed FP32); the FP32 class kernels are in
// phmm_fwd32.cuh, instantiated per mode in phmm_fwd32_m0/m1/m2.cu.
//
// Every kernel class (precision, rows per lane, variant, FP32 gap-parameter mode, stripe mode) is
// its own kernel, so each gets the register allocation its own live state needs instead of the
// union of all paths.  Work items are grouped by class on the host.
#include <cuda_runtime.h>

#include "phmm_fwd32.cuh"
#include "phmm_warp64.cuh"
#include "phmm_kernels.h"

namespace phmm {

// ------------------------------------------------------------------------------------------
// Before the passes (grid-stride): haplotype bytes -> per-variant match codes, and the output reset:
// every likelihood NaN (pairs with an empty read or haplotype stay NaN), flags 0.  One launch for both: a
// small batch waits for each (about 3 us), and a large one streams both through HBM either way.
// ------------------------------------------------------------------------------------------
__global__ void prep_kernel(const BatchDesc* __restrict__ desc, const uint8_t* __restrict__ hap_bases,
                            uint32_t* __restrict__ codes_inter, uint32_t* __restrict__ codes_intra,
                            double* __restrict__ out, uint8_t* __restrict__ flags)
{
    const uint64_t total = desc->hap_bases_total;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t i = first; i < total; i += stride) {
        const uint8_t b = hap_bases[i];
        codes_inter[kCodePad + i] = hap_code(b, kInter);
        codes_intra[kCodePad + i] = hap_code(b, kIntra);
    }
    // guard codes on both sides of the stream: match nothing
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k < kCodePad; k += blockDim.x) {
            codes_inter[k] = 0u;
            codes_intra[k] = 0u;
            codes_inter[kCodePad + total + k] = 0u;
            codes_intra[kCodePad + total + k] = 0u;
        }
    }
    const uint64_t outs = desc->out_total;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    for (uint64_t i = first; i < outs; i += stride) {
        out[i] = nan;
        if (flags) flags[i] = 0;
    }
}

// ------------------------------------------------------------------------------------------
// FP64 pass for one class over the runs of underflowed pairs the FP32 pass appended, one run per
// claim, streamed through the read like an FP32 work item.
// ------------------------------------------------------------------------------------------
// Resident warps per SM of the FP64 classes of mode 0 (constant gaps, insertion = deletion), the
// compiler's register bound: 16 (128 registers; up to 200 bytes of spill loads) for 8 and 7 rows per lane in
// one stripe, 12 (168 registers, no spills) for stripes.  Measured on B200 with the unflushed sweep, 8 rows:
// the FP64 pass of 60 low-quality regions 22.6 ms at 16 warps, 23.0 at 12, 23.6 at 11; of the 1,000-region
// batch 4.54 and 4.63 ms at 16 and 12; 7 rows 2.80 ms at 16 and 2.87 at 12; stripes: a call of 24 regions of
// long reads 9.71 ms at 16 and 9.47 at 12, and of 11,520 pairs of foreign long reads, all swept with
// flushes, 34.1 and 31.0 ms.  The other classes keep what they need.  Build-time settings.
#ifndef PHMM_F64_MIN_WARPS_K8
#define PHMM_F64_MIN_WARPS_K8 16
#endif
#ifndef PHMM_F64_MIN_WARPS_K7
#define PHMM_F64_MIN_WARPS_K7 16
#endif
#ifndef PHMM_F64_MIN_WARPS_MULTI
#define PHMM_F64_MIN_WARPS_MULTI 12
#endif
template <int K, int PM, bool MULTI>
constexpr int min_blocks64()
{
    return PM != PM_EQ ? 1 : MULTI ? PHMM_F64_MIN_WARPS_MULTI : K == 8 ? PHMM_F64_MIN_WARPS_K8 : K == 7 ? PHMM_F64_MIN_WARPS_K7 : 1;
}

// UNF: the all-FP64 check arithmetic (plain multiply and add), used to measure the error of every
// likelihood; the recompute pass proper uses the reference's contracted arithmetic.
template <int K, int V, int PM, bool MULTI, bool UNF = false>
__global__ void __launch_bounds__(kFwdBlock, min_blocks64<K, PM, MULTI>()) fwd_f64_kernel(BatchView b, ProbTables<double> tb, PassControl pc)
{
    __shared__ PriorTable64<K> tab;
    const int lane = threadIdx.x & (kWarp - 1);
    const unsigned int warp_id = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
    warp_reruns64<K, V, PM, MULTI, UNF>(b, tb, pc, tab.v, lane, warp_id);
}

// ------------------------------------------------------------------------------------------
// FP32 FMA throughput probe: 16 independent FMA chains per thread on every SM.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) fma_peak_kernel(float* sink, int iters, float a, float b)
{
    float x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = (float)(threadIdx.x + k) * 1e-3f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = __fmaf_rn(x[k], a, b);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += x[k];
    if (s == -1.0f) sink[blockIdx.x] = s;  // never true; keeps the chains alive
}

// Same with packed FFMA2: 16 independent float2 chains (32 FMAs per thread per iteration).
__global__ void __launch_bounds__(256) fma2_peak_kernel(float* sink, int iters, float a, float b)
{
    float2 x[16];
    const float2 a2 = make_float2(a, a), b2 = make_float2(b, b);
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = make_float2((float)(threadIdx.x + k) * 1e-3f, (float)(threadIdx.x - k) * 1e-3f);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = __ffma2_rn(x[k], a2, b2);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += x[k].x + x[k].y;
    if (s == -1.0f) sink[blockIdx.x] = s;
}

cudaError_t launch_fma_peak(float* sink, int blocks, int iters, bool packed, cudaStream_t st)
{
    if (packed)
        fma2_peak_kernel<<<blocks, 256, 0, st>>>(sink, iters, 0.999f, 1e-4f);
    else
        fma_peak_kernel<<<blocks, 256, 0, st>>>(sink, iters, 0.999f, 1e-4f);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------
// Class tables and host-side launch wrappers.
// ------------------------------------------------------------------------------------------
typedef void (*F64Kernel)(BatchView, ProbTables<double>, PassControl);

#define PHMM_ROW64(V, PM)                                                                                 \
    fwd_f64_kernel<1, V, PM, false>, fwd_f64_kernel<2, V, PM, false>, fwd_f64_kernel<3, V, PM, false>,    \
        fwd_f64_kernel<4, V, PM, false>, fwd_f64_kernel<5, V, PM, false>, fwd_f64_kernel<6, V, PM, false>, \
        fwd_f64_kernel<7, V, PM, false>, fwd_f64_kernel<8, V, PM, false>, fwd_f64_kernel<8, V, PM, true>

static const F64Kernel kF64[kClasses64] = {PHMM_ROW64(kInter, PM_EQ), PHMM_ROW64(kInter, PM_ROW),
                                           PHMM_ROW64(kIntra, PM_ROW)};

// All-FP64 check kernels: the same shapes with plain multiply/add, per-row gap parameters (any
// read), inter and intra variants (FP64 classes of modes 1 and 2).
#define PHMM_ROW64_CHECK(V)                                                                               \
    fwd_f64_kernel<1, V, PM_ROW, false, true>, fwd_f64_kernel<2, V, PM_ROW, false, true>,                 \
        fwd_f64_kernel<3, V, PM_ROW, false, true>, fwd_f64_kernel<4, V, PM_ROW, false, true>,             \
        fwd_f64_kernel<5, V, PM_ROW, false, true>, fwd_f64_kernel<6, V, PM_ROW, false, true>,             \
        fwd_f64_kernel<7, V, PM_ROW, false, true>, fwd_f64_kernel<8, V, PM_ROW, false, true>,             \
        fwd_f64_kernel<8, V, PM_ROW, true, true>
static const F64Kernel kF64Check[2 * 9] = {PHMM_ROW64_CHECK(kInter), PHMM_ROW64_CHECK(kIntra)};

cudaError_t launch_prep(const BatchDesc* desc, const uint8_t* hap_bases, uint32_t* codes_inter, uint32_t* codes_intra,
                        double* out, uint8_t* flags, int num_sms, cudaStream_t st)
{
    prep_kernel<<<num_sms * 8, 256, 0, st>>>(desc, hap_bases, codes_inter, codes_intra, out, flags);
    return cudaGetLastError();
}

cudaError_t launch_fwd(int precision, int cls, const BatchView& b, const ProbTables<float>& tf,
                       const ProbTables<double>& td, const PassControl& pc, int grid, cudaStream_t st)
{
    if (cls < 0 || cls >= (precision == 32 ? kClasses32 : kClasses64) || grid <= 0) return cudaErrorInvalidValue;
    if (precision == 32) {
        const int mode = cls / kShapes32, shape = cls % kShapes32;
        if (mode == 0) return launch_f32_mode0(shape, b, tf, pc, grid, st);
        if (mode == 1) return launch_f32_mode1(shape, b, tf, pc, grid, st);
        return launch_f32_mode2(shape, b, tf, pc, grid, st);
    }
    kF64[cls]<<<grid, kFwdBlock, 0, st>>>(b, td, pc);
    return cudaGetLastError();
}

cudaError_t launch_f64_check(int cls, const BatchView& b, const ProbTables<double>& td, const PassControl& pc, int grid,
                             cudaStream_t st)
{
    if (cls < 9 || cls >= kClasses64 || grid <= 0) return cudaErrorInvalidValue;
    kF64Check[cls - 9]<<<grid, kFwdBlock, 0, st>>>(b, td, pc);
    return cudaGetLastError();
}

cudaError_t occupancy_f64_check(int cls, int* blocks_per_sm)
{
    if (cls < 9 || cls >= kClasses64) return cudaErrorInvalidValue;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kF64Check[cls - 9], kFwdBlock, 0);
}

cudaError_t occupancy(int precision, int cls, int* blocks_per_sm)
{
    if (cls < 0 || cls >= (precision == 32 ? kClasses32 : kClasses64)) return cudaErrorInvalidValue;
    if (precision == 32) {
        const int mode = cls / kShapes32, shape = cls % kShapes32;
        if (mode == 0) return occupancy_f32_mode0(shape, blocks_per_sm);
        if (mode == 1) return occupancy_f32_mode1(shape, blocks_per_sm);
        return occupancy_f32_mode2(shape, blocks_per_sm);
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kF64[cls], kFwdBlock, 0);
}

}  // namespace phmm
