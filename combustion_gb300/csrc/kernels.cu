// Plain FP64 kernels: species production rates (reaction.rs:207-391), per-reaction rates of progress
// (reaction.rs:329-354) and mixture-averaged transport (transport.rs:141-210), one cell per thread.
//
// Every thread of a warp walks the same reaction / species / pair at the same time, so each table read
// is a broadcast; the per-cell working arrays (concentrations, Gibbs exponentials, accumulators) live in
// thread-local memory. The FP64 pipe is the bottleneck; nothing else here comes close to its limits.
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "device_math.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "rates_cell.cuh"
#include "tables.h"
#include "transport_cell.cuh"

namespace cbg {

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(kBlock) rates_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                      const __grid_constant__ RatesArgs<KMAX> io, size_t n,
                                                      int* status) {
    let_next_start();
    __shared__ uint64_t bar;
    const uint8_t* tab = gtab;
    if (SMEM) {  // the whole blob, math tables first, into dynamic shared memory
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
        tab = cb_dsmem;
    } else {  // tables read from global memory; only the math tables go to shared memory
        load_math(gtab);
    }
    const RatesTables tb(tab);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        rates_cell<KMAX>(tb, io, i);
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(kBlock) reaction_rates_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                               const __grid_constant__ ReactionRatesArgs<KMAX> io,
                                                               size_t n, int* status) {
    __shared__ uint64_t bar;
    const uint8_t* tab = gtab;
    if (SMEM) {  // the whole blob, math tables first, into dynamic shared memory
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
        tab = cb_dsmem;
    } else {  // tables read from global memory; only the math tables go to shared memory
        load_math(gtab);
    }
    const RatesTables tb(tab);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        reaction_rates_cell<KMAX>(tb, io, i);
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(kTransportBlock) transport_kernel(const uint8_t* __restrict__ gtab, uint32_t tab_bytes,
                                                          const __grid_constant__ TransportArgs<KMAX> io,
                                                          size_t n, int* status) {
    const EndAfterPrevious last;
    __shared__ uint64_t bar;
    const uint8_t* tab = gtab;
    if (SMEM) {  // the whole blob, math tables first, into dynamic shared memory
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
        tab = cb_dsmem;
    } else {  // tables read from global memory; only the math tables go to shared memory
        load_math(gtab);
    }
    if (io.count) n = min(n, (size_t)*io.count);  // gathered cells: the count is known on the device only
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (size_t)gridDim.x * blockDim.x) {
        const size_t i = io.index ? (size_t)(io.index[j] & kIndexMask) : j;
        transport_cell<KMAX>(tab, io, i, (io.flags & kCompactOut) ? j : i);
    }
}

template <int KMAX, bool SMEM>
__global__ void __launch_bounds__(32 * kWarpCellWarps) transport_warp_kernel(const uint8_t* __restrict__ gtab,
                                                                           uint32_t tab_bytes,
                                                                           const __grid_constant__ TransportArgs<KMAX> io,
                                                                           size_t n, int* status) {
    const EndAfterPrevious last;
    __shared__ uint64_t bar;
    const uint8_t* tab = gtab;
    if (SMEM) {
        if (!stage_to_shared(cb_dsmem, gtab, tab_bytes, &bar, status)) return;
        tab = cb_dsmem;
    } else {
        load_math(gtab);
    }
    const size_t table_bytes = warp_table_bytes(SMEM, tab_bytes);
    double* sh = reinterpret_cast<double*>(cb_dsmem + table_bytes) + (size_t)(threadIdx.x >> 5) * kWarpScratch<KMAX>;
    if (io.count) n = min(n, (size_t)*io.count);
    const size_t warps = (size_t)gridDim.x * kWarpCellWarps;
    for (size_t j = (size_t)blockIdx.x * kWarpCellWarps + (threadIdx.x >> 5); j < n; j += warps) {
        const size_t i = io.index[j] & kIndexMask;
        transport_cell_warp<KMAX>(tab, io, i, (io.flags & kCompactOut) ? j : i, sh);
    }
}

// ---------------------------------------------------------------------------------------------------
// Non-finite values by exponent bits (all ones): integer instructions only.
__global__ void count_nonfinite_kernel(const __grid_constant__ CountArgs args, size_t n, unsigned long long* count) {
    unsigned long long c = 0;
    for (int q = 0; q < args.m; q++)
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
            c += (__double2hiint(args.a[q][i]) & 0x7ff00000) == 0x7ff00000;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

cudaError_t launch_count_nonfinite(const CountArgs& args, size_t n, unsigned long long* count, cudaStream_t st) {
    if (n == 0 || args.m == 0) return cudaSuccess;
    size_t grid = (n + 255) / 256;
    if (grid > (size_t)sm_count() * 8) grid = (size_t)sm_count() * 8;
    count_nonfinite_kernel<<<(unsigned)grid, 256, 0, st>>>(args, n, count);
    return cudaGetLastError();
}

// The elementary functions of the plain path on device arrays (which: 0 exp, 1 log, 2 reciprocal), for
// accuracy checks against CUDA's own functions.
__global__ void math_check_kernel(const uint8_t* math, int which, const double* x, double* y, size_t n) {
    load_math(math);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = x[i];
        y[i] = which == 0 ? exp64(v) : which == 1 ? log64(v) : rcp64(v);
    }
}

cudaError_t launch_math_check(const uint8_t* math, int which, const double* x, double* y, size_t n,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    size_t grid = (n + 255) / 256;
    if (grid > 4096) grid = 4096;
    math_check_kernel<<<(unsigned)grid, 256, kMathBytes, st>>>(math, which, x, y, n);
    return cudaGetLastError();
}

// Test hook: polls of the first staging wait of the plain kernels (negative: the default limit).
cudaError_t set_stage_wait_polls(long long polls) {
    const long long v = polls < 0 ? kWaitLimit : polls;
    const cudaError_t e = cudaMemcpyToSymbol(g_stage_wait_polls, &v, sizeof v);
    const cudaError_t e2 = e == cudaSuccess ? set_stage_wait_polls_x(v) : e;
    return e2 == cudaSuccess ? set_stage_wait_polls_tx(v) : e2;
}

int max_table_smem() {
    static int v = -1;
    if (v < 0) {
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        v = optin - 1024;  // room for the static shared variables
    }
    return v;
}

CB_DISPATCH(launch_rates, rates_kernel, RatesArgs, kBlock, kMathBytes, false)
CB_DISPATCH(launch_reaction_rates, reaction_rates_kernel, ReactionRatesArgs, kBlock, kMathBytes, false)

CB_WAVE(wave_rates, rates_kernel, kBlock, kMathBytes)
CB_WAVE(wave_reaction_rates, reaction_rates_kernel, kBlock, kMathBytes)
CB_WAVE(wave_transport, transport_kernel, kTransportBlock, kMathBytes)

namespace {
// Gathered launches of up to this many cells per SM go warp-per-cell (above 16 species): one cell per
// thread would leave most SMs idle and the rest latency-bound; beyond it, one per thread keeps every
// lane busy without the warp form's serial chains.
constexpr size_t kWarpCellsPerSm = 128;

template <int KMAX>
cudaError_t launch_transport_k(const uint8_t* tab, uint32_t tab_bytes, const TransportArgs<KMAX>& io, size_t n,
                               cudaStream_t st, int* status) {
    if constexpr (KMAX >= 64) {
        if (io.index && n <= (size_t)sm_count() * kWarpCellsPerSm) {
            const size_t scratch = (size_t)kWarpCellWarps * kWarpScratch<KMAX> * sizeof(double);
            const bool smem = warp_table_bytes(true, tab_bytes) + scratch <= (size_t)max_table_smem();
            const size_t bytes = warp_table_bytes(smem, tab_bytes) + scratch;
            auto kern = smem ? transport_warp_kernel<KMAX, true> : transport_warp_kernel<KMAX, false>;
            const cudaError_t e = allow_shared(kern);
            if (e != cudaSuccess) return e;
            int per_sm = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kWarpCellWarps, bytes);
            if (per_sm < 1) per_sm = 1;
            size_t grid = (size_t)sm_count() * per_sm;
            const size_t want = (n + kWarpCellWarps - 1) / kWarpCellWarps;
            if (want < grid) grid = want ? want : 1;
            kern<<<(unsigned)grid, 32 * kWarpCellWarps, bytes, st>>>(tab, tab_bytes, io, n, status);
            return cudaGetLastError();
        }
    }
    return launch_table_kernel<kTransportBlock>(transport_kernel<KMAX, true>, transport_kernel<KMAX, false>, tab,
                                                tab_bytes, io, n, kMathBytes, true, st, status);
}
}  // namespace

cudaError_t launch_transport(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                             cudaStream_t st, int* status) {
    switch (kmax) {
    case 16: return launch_transport_k<16>(tab, tab_bytes, *static_cast<const TransportArgs<16>*>(args), n, st, status);
    case 64: return launch_transport_k<64>(tab, tab_bytes, *static_cast<const TransportArgs<64>*>(args), n, st, status);
    case 256:
        return launch_transport_k<256>(tab, tab_bytes, *static_cast<const TransportArgs<256>*>(args), n, st, status);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace cbg
