// Kernel arguments and launchers shared by the C ABI (capi.cu) and the kernels (kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cbg {

// Threads per block. Each block stages its own copy of the tables in shared memory, which shares the
// SM's 256 KB with the L1 cache that holds the thread-local arrays (concentrations, Gibbs exponentials,
// accumulators); 768-thread blocks keep one or two copies per SM instead of two or three and leave L1
// that room: measured at K = 53, 2^22 cells, the mixed rates kernel 54.2 -> 38.1 ms (256-thread blocks
// before; 1024-thread blocks 45.5 ms), the FP64 rates kernel 119.6 -> 117.0 ms, mixed transport
// 1 ms faster. FP64 transport (tables of 135 KB, one block per SM) keeps 256 threads: 768 ran no
// faster (the FP64 pipe is 97 % busy either way) and its per-thread arrays then spilled past L1 into
// DRAM (24 KB per cell instead of 2 KB).
constexpr int kBlock = 768;
// The fixed-point rates kernels are bound by latency (integer chains, thread-local arrays in L2) as much as by
// a pipe: 1,024 threads (64 registers) 40.2 ms, 768 (80) 48.0 ms at 2^22 cells of 53 species.
constexpr int kRatesXBlock = 1024;
// Fixed-point transport, 2^22 cells: 53 species 45.1 ms with 512 threads (128 registers, Wilke rows without spills),
// 48.3 with 640; 10 species 2.95 ms with 512, 2.80 with 768; 250 species (131,072 cells), whose arrays are in L2
// either way, 50 ms with 512 and 40 with 1,024.
template <int KMAX>
constexpr int kTransportXBlock = KMAX == 16 ? 768 : KMAX == 64 ? 512 : 1024;
constexpr int kTransportBlock = 256;
constexpr int kTransportMixedBlock = 768;

// One pointer per input / output array (struct of arrays), passed by value as a kernel parameter.
template <int KMAX>
struct RatesArgs {
    const double* in[KMAX + 3];  // P/R, R/P, T, V, n_0 .. n_{K-2}
    double* out[KMAX + 2];       // dT/dt, dV/dt, wdot_0 .. wdot_{A-1}
    uint32_t flags;              // bit 1: P/R and R/P are single values
    const uint8_t* f64_tab;      // fixed-point kernels: the FP64 tables, in global memory
};

// Per-reaction rates of progress: inputs P/R, T, V, n_0 .. n_{K-2}; one output per reaction.
constexpr int kMaxReactions = 2048;
template <int KMAX>
struct ReactionRatesArgs {
    const double* in[KMAX + 2];
    double* out[kMaxReactions];
    uint32_t flags;
    const uint8_t* f64_tab;
};

// Transport input layouts: the reference's (sum n, T/T0, n...) or, with kFromRates, the rates inputs
// (P/R, R/P, T, V, n...) from which sum n = (P/R * V) / T and T/T0 are derived per cell.
constexpr uint32_t kUniformPressure = 2u;
constexpr uint32_t kFromRates = 4u;
// Gathered cells (the transport surrogate's fallback and audit): cell j of the launch is input cell
// index[j] & kIndexMask, its outputs go to that cell too or, with kCompactOut, to position j.
constexpr uint32_t kCompactOut = 8u;
// The launch may start while the kernel before it on the stream still runs (device_common.cuh).
constexpr uint32_t kOverlap = 16u;
constexpr uint32_t kIndexMask = 0x7fffffffu;

template <int KMAX>
struct TransportArgs {
    const double* in[KMAX + 3];  // sum n, T/T0, n_0 .. n_{K-2} (or the rates inputs with kFromRates)
    double* out[KMAX + 2];       // lambda/lambda0, mu/mu0, rhoD_k/mu0
    uint32_t flags;
    const uint32_t* index;       // gathered cells (null: cell j is input j)
    const uint32_t* count;       // number of gathered cells, read on the device (null: n)
    const uint8_t* f64_tab;      // fixed-point kernels: the FP64 tables, in global memory
    // A second list behind the n1 cells of `index` (one cell per warp only): its outputs go to position j of
    // out2 + k stride2.
    const uint32_t* index2;
    double* out2;
    size_t n1, stride2;
};

// Smallest compiled capacity holding K species (0 if none).
// (The per-cell efficiency sums of up to 4 * KMAX third-body / falloff reactions are kept per thread.)
inline int kmax_for(int K, int n_eff) {
    for (int km : {16, 64, 256})
        if (K <= km && n_eff <= 4 * km) return km;
    return 0;
}

int max_table_smem();
cudaError_t set_stage_wait_polls(long long polls);
// The same of the fixed-point kernels' translation units.
cudaError_t set_stage_wait_polls_x(long long polls);
cudaError_t set_stage_wait_polls_tx(long long polls);

// Non-finite values (NaN, infinity) in up to kCountArrays arrays of n doubles, added to *count.
constexpr int kCountArrays = 512;
struct CountArgs {
    const double* a[kCountArrays];
    int m;
};
cudaError_t launch_count_nonfinite(const CountArgs& args, size_t n, unsigned long long* count, cudaStream_t st);

// A kernel's limit of dynamic shared memory, raised to the device's. The limit belongs to the process: with what a call
// needs in its place, a call of another host thread could lower it between this one's setting and its launch.
template <class K>
cudaError_t allow_shared(K kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_table_smem());
}

// Blocks of a persistent table kernel resident per SM, the tables in shared memory (smem: the variant
// ksmem, whose dynamic shared memory limit is raised first) or read from global memory (kglobal, only
// the math tables in shared memory).
template <class KS, class KG>
cudaError_t table_kernel_occupancy(KS ksmem, KG kglobal, int block, uint32_t tab_bytes, uint32_t math_bytes,
                                   bool smem, int* per_sm) {
    *per_sm = 1;
    if (smem) {
        cudaError_t e = allow_shared(ksmem);
        // the split of shared memory and L1 that an earlier call asked for (set_carveout) is not this call's
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(ksmem, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutDefault);
        if (e != cudaSuccess) return e;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, ksmem, block, tab_bytes);
    } else {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kglobal, block, math_bytes);
    }
    if (*per_sm < 1) *per_sm = 1;
    return cudaSuccess;
}

// Shared memory (of an SM's 256 KB, shared with L1) for `per_sm` resident blocks of a table kernel, whatever
// block size a launch takes. The preference stays with the kernel: table_kernel_occupancy takes it back for the next
// call (left from a call of a smaller mechanism, 2^20 cells of mixed rates at 53 species took 11.5 ms, 9.4 without).
template <class K>
cudaError_t set_carveout(K kernel, int per_sm, uint32_t bytes) {
    const int most = max_table_smem() + 1024, want = per_sm * (int)(bytes + 2048);
    const int percent = want >= most ? 100 : (int)((100ll * want + most - 1) / most);
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent);
}

// Cells one wave of a kernel's persistent grid covers (its threads resident on the whole GPU): every
// thread of a launch over a multiple of it gets the same number of cells. Host arrays go through the
// GPU in chunks of whole waves.
size_t wave_rates(int kmax, uint32_t tab_bytes);
size_t wave_reaction_rates(int kmax, uint32_t tab_bytes);
size_t wave_transport(int kmax, uint32_t tab_bytes);
size_t wave_rates_mixed(int kmax, uint32_t tab_bytes);
size_t wave_transport_mixed(int kmax, uint32_t tab_bytes);
cudaError_t launch_math_check(const uint8_t* math, int which, const double* x, double* y, size_t n,
                              cudaStream_t st);
cudaError_t launch_rates(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                         cudaStream_t st, int* status);
cudaError_t launch_reaction_rates(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                  cudaStream_t st, int* status);
// The fixed-point functions on doubles: `tab` [MathTables][FixMath].
cudaError_t launch_fixed_math_check(const uint8_t* tab, int which, const double* x, double* y, size_t n, cudaStream_t st);
// The fixed-point forms (kernels_fixed.cu); `args` carries the FP64 tables as well.
// warp_bytes: a warp's scratch in the form of one cell per warp (rates_warp_bytes).
cudaError_t launch_rates_x(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n, size_t warp_bytes,
                           cudaStream_t st, int* status);
cudaError_t launch_reaction_rates_x(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                    size_t warp_bytes, cudaStream_t st, int* status);
inline size_t rates_warp_bytes(int K, int R, int n_eff) { return (4 * (size_t)K + (size_t)n_eff + (size_t)R) * sizeof(double); }
cudaError_t launch_transport_x(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                               cudaStream_t st, int* status);
size_t wave_transport_x(int kmax, uint32_t tab_bytes);
size_t transport_x_warp_cells(int kmax);  // most cells of a call that goes one cell per warp
size_t wave_rates_x(int kmax, uint32_t tab_bytes);
size_t wave_reaction_rates_x(int kmax, uint32_t tab_bytes);
// warp_bytes as above: small calls go one cell per warp (mixed_warp.cu); `tab_bytes` is what the kernels stage, the
// species' reaction lists follow.
cudaError_t launch_rates_mixed(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                               size_t warp_bytes, cudaStream_t st, int* status);
cudaError_t launch_rates_mixed_warp(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                    size_t warp_bytes, cudaStream_t st, int* status);
cudaError_t launch_transport_mixed_warp(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                        cudaStream_t st, int* status);
cudaError_t launch_transport_mixed(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                                   cudaStream_t st, int* status);
cudaError_t launch_transport(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n,
                             cudaStream_t st, int* status);

}  // namespace cbg
