// Launch of the table kernels: persistent grids, tables in shared memory when they fit.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"

namespace cbg {

inline int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    return sms;
}

template <class Args>
bool gathered(const Args&) { return false; }
template <int KMAX>
bool gathered(const TransportArgs<KMAX>& io) { return io.index != nullptr; }

template <class Args>
bool overlapped(const Args&) { return false; }
template <int KMAX>
bool overlapped(const TransportArgs<KMAX>& io) { return io.flags & kOverlap; }

template <class K, class Args>
cudaError_t launch_one(K kernel, size_t grid, int block, size_t bytes, cudaStream_t st, const uint8_t* tab, uint32_t tab_bytes,
                       const Args& io, size_t n, int* status) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = overlapped(io) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, tab, tab_bytes, io, n, status);
}

// Persistent grid: as many blocks as fit on the GPU at once (each stages the tables once). A call of at most
// two waves takes smaller blocks, so that every SM gets the same share of each wave and small calls spread
// over all of them: blocks of 768 left 10,100 cells on 14 SMs. (Beyond two waves the last one weighs less
// than the warps that smaller blocks leave out: mixed rates of 2.5 waves ran 8 % slower.) The shared-memory
// carve-out stays that of the full blocks: the driver would size it for as many small blocks as fit, at the
// expense of the L1 that holds the thread-local arrays.
// Gathered cells of less than a wave (a trust gate's fallback or audit, whose number may be known on the
// device only) go in one-warp blocks.
// Without room in shared memory the tables are read through L1/L2 (kglobal, `math_bytes` staged).
template <int BLOCK, class Args, class KS, class KG>
cudaError_t launch_table_kernel(KS ksmem, KG kglobal, const uint8_t* tab, uint32_t tab_bytes, const Args& io,
                                size_t n, uint32_t math_bytes, bool one_warp_if_gathered, cudaStream_t st, int* status) {
    const bool smem = (int)tab_bytes <= max_table_smem();
    int block = BLOCK, per_sm = 1;
    cudaError_t e = table_kernel_occupancy(ksmem, kglobal, BLOCK, tab_bytes, math_bytes, smem, &per_sm);
    if (e != cudaSuccess) return e;
    size_t grid = (size_t)sm_count() * per_sm;
    if (gathered(io)) {
        if (one_warp_if_gathered || n < grid * BLOCK) {
            block = 32;
            e = table_kernel_occupancy(ksmem, kglobal, block, tab_bytes, math_bytes, smem, &per_sm);
            if (e != cudaSuccess) return e;
            grid = (size_t)sm_count() * per_sm;
        }
    } else if (n <= 2 * grid * BLOCK) {
        const size_t waves = (n + grid * BLOCK - 1) / (grid * BLOCK), share = (n + waves * grid - 1) / (waves * grid);
        block = (int)((share + 31) / 32 * 32);
        if (smem) e = set_carveout(ksmem, per_sm, tab_bytes);
        if (e != cudaSuccess) return e;
    }
    const size_t want = (n + block - 1) / block;
    if (want < grid) grid = want ? want : 1;
    return smem ? launch_one(ksmem, grid, block, tab_bytes, st, tab, tab_bytes, io, n, status)
                : launch_one(kglobal, grid, block, math_bytes, st, tab, tab_bytes, io, n, status);
}

// One cell per warp, up to WARPS of them in a block: as many warps as fit beside the tables (or, of a large mechanism, beside the functions' tables).
template <int WARPS, class KS, class KG, class Args>
cudaError_t launch_warp_kernel(KS ksmem, KG kglobal, const uint8_t* tab, uint32_t tab_bytes, const Args& io, size_t n,
                               uint32_t math, size_t warp_bytes, cudaStream_t st, int* status) {
    const size_t share = (n + sm_count() - 1) / sm_count();
    const bool smem = tab_bytes + 2 * warp_bytes <= (size_t)max_table_smem();
    int warps = share < (size_t)WARPS ? (int)share : WARPS;
    while (warps > 1 && (smem ? tab_bytes : math) + warps * warp_bytes > (size_t)max_table_smem()) warps--;
    const size_t bytes = (smem ? tab_bytes : math) + warps * warp_bytes;
    if (bytes > (size_t)max_table_smem()) return cudaErrorInvalidConfiguration;
    const cudaError_t e = smem ? allow_shared(ksmem) : allow_shared(kglobal);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    if (smem) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ksmem, 32 * warps, bytes);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kglobal, 32 * warps, bytes);
    if (per_sm < 1) per_sm = 1;
    size_t grid = (size_t)sm_count() * per_sm;
    const size_t want = (n + warps - 1) / warps;
    if (want < grid) grid = want ? want : 1;
    return smem ? launch_one(ksmem, grid, 32 * warps, bytes, st, tab, tab_bytes, io, n, status)
                : launch_one(kglobal, grid, 32 * warps, bytes, st, tab, tab_bytes, io, n, status);
}

// One cell per block of TEAM warps, for calls of at most a cell per SM.
constexpr int kTeamWarps = 8;
template <int TEAM, class KS, class KG, class Args>
cudaError_t launch_team_kernel(KS ksmem, KG kglobal, const uint8_t* tab, uint32_t tab_bytes, const Args& io, size_t n,
                               uint32_t math, size_t cell_bytes, cudaStream_t st, int* status) {
    const bool smem = tab_bytes + cell_bytes <= (size_t)max_table_smem();
    const size_t bytes = (smem ? tab_bytes : math) + cell_bytes, grid = n ? n : 1;
    const cudaError_t e = smem ? allow_shared(ksmem) : allow_shared(kglobal);
    if (e != cudaSuccess) return e;
    return smem ? launch_one(ksmem, grid, 32 * TEAM, bytes, st, tab, tab_bytes, io, n, status)
                : launch_one(kglobal, grid, 32 * TEAM, bytes, st, tab, tab_bytes, io, n, status);
}

template <int BLOCK, class KS, class KG>
size_t wave_of(KS ksmem, KG kglobal, uint32_t tab_bytes, uint32_t math_bytes) {
    int per_sm = 1;
    if (table_kernel_occupancy(ksmem, kglobal, BLOCK, tab_bytes, math_bytes, (int)tab_bytes <= max_table_smem(),
                               &per_sm) != cudaSuccess)
        return 0;
    return (size_t)sm_count() * per_sm * BLOCK;
}

#define CB_DISPATCH(FN, KERNEL, ARGS, BLOCK, MATH, ONE_WARP)                                                       \
    cudaError_t FN(int kmax, const uint8_t* tab, uint32_t tab_bytes, const void* args, size_t n, cudaStream_t st, \
                   int* status) {                                                                                 \
        switch (kmax) {                                                                                           \
        case 16: return launch_table_kernel<BLOCK>(KERNEL<16, true>, KERNEL<16, false>, tab, tab_bytes,           \
                                                   *static_cast<const ARGS<16>*>(args), n, MATH, ONE_WARP, st, status);     \
        case 64: return launch_table_kernel<BLOCK>(KERNEL<64, true>, KERNEL<64, false>, tab, tab_bytes,           \
                                                   *static_cast<const ARGS<64>*>(args), n, MATH, ONE_WARP, st, status);     \
        case 256: return launch_table_kernel<BLOCK>(KERNEL<256, true>, KERNEL<256, false>, tab, tab_bytes,        \
                                                    *static_cast<const ARGS<256>*>(args), n, MATH, ONE_WARP, st, status);   \
        default: return cudaErrorInvalidValue;                                                                    \
        }                                                                                                         \
    }

#define CB_WAVE(FN, KERNEL, BLOCK, MATH)                                                         \
    size_t FN(int kmax, uint32_t tab_bytes) {                                                    \
        switch (kmax) {                                                                          \
        case 16: return wave_of<BLOCK>(KERNEL<16, true>, KERNEL<16, false>, tab_bytes, MATH);    \
        case 64: return wave_of<BLOCK>(KERNEL<64, true>, KERNEL<64, false>, tab_bytes, MATH);    \
        case 256: return wave_of<BLOCK>(KERNEL<256, true>, KERNEL<256, false>, tab_bytes, MATH); \
        default: return 0;                                                                       \
        }                                                                                        \
    }

}  // namespace cbg
