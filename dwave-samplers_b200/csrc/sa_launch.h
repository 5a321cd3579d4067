// Launch helpers for the sweep kernels (implemented in sa_launch.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "sa_types.h"

namespace b200sa {

constexpr int kMaxThreadsPerCta = 512;
// Register budgets of the sweep kernels (per thread): 128 (launch bounds of
// 512 threads, one CTA), kRegs80 and kRegs64.
constexpr int kRegs80 = 80;
constexpr int kRegs64 = 64;
constexpr int kRegClasses = 3;  // 0: 128, 1: 80, 2: 64

// Kernel kind: bit 0 Gibbs, bit 1 random order, bit 2 in-window resolution
// (sequential order only; ProblemDev::resolve), bit 3 state in registers
// (ProblemDev::dense; both orders, without bit 2).
constexpr int kKindGibbs = 1;
constexpr int kKindRandom = 2;
constexpr int kKindResolve = 4;
constexpr int kKindDense = 8;
// Bit 4 equal list lengths (ProblemDev::regular_degree; without bit 3; the
// two kinds of lists have kernels of their own, each with its path's registers
// and code alone: uneven batch 93.6 -> 88.6 ms, 50 reads of a sparse n = 20011
// problem 26.1 -> 23.6, n = 1000, 1000 reads 4.7 -> 4.2).
constexpr int kKindRegular = 16;
constexpr int kNumKinds = 32;

// Kernels with the state in registers: 1, 2, 4, 8 or kDenseSlots variables per
// lane by the launch's largest n, one register budget each.
inline int dense_slots(int max_n) {
    return max_n <= 32 ? 0 : max_n <= 64 ? 1 : max_n <= 128 ? 2 : max_n <= 256 ? 3 : 4;
}
inline int dense_reg_class(int max_n) { return max_n <= 64 ? 2 : max_n <= 128 ? 1 : 0; }

// Kernel variant: bits 0-4 kind, bits 5-6 state location (kStageGlobal,
// kStageShared, kStageSpins, kStageBand), bits 7-8 register class (0: 128, 1:
// 80, 2: 64 registers), bits 9-11 dense_slots of kinds with the state in
// registers.
inline int kernel_variant(int kind, int stage, int reg_class = 0, int max_n = 0) {
    return (kind & (kNumKinds - 1)) | (stage << 5) | (reg_class << 7) |
           ((kind & kKindDense) ? dense_slots(max_n) << 9 : 0);
}
inline int variant_stage(int variant) { return (variant >> 5) & 3; }
inline int variant_reg_class(int variant) { return (variant >> 7) & 3; }
inline int variant_slots(int variant) { return variant >> 9; }

// Bytes of the touch bitmap of a launch (random order outside registers).
inline int kind_touch_bytes(int kind, int max_n) {
    return touch_bytes_for((kind & kKindRandom) && !(kind & kKindDense), max_n);
}

cudaError_t upload_jump_table(const uint32_t table[][4], cudaStream_t stream);
cudaError_t scatter_weights(double *arena, const int64_t *dst, const int32_t *src, int64_t num_j,
                            int64_t total, const double *J, const double *h,
                            cudaStream_t stream);
cudaError_t launch_sa(int variant, const LaunchArgs &args, int grid, int warps_per_cta,
                      int region_bytes, cudaStream_t stream);
cudaError_t kernel_occupancy(int variant, int warps_per_cta, int region_bytes,
                             int *ctas_per_sm);
cudaError_t launch_sd(bool sparse, bool smem, bool flat, const SdArgs &args, int grid,
                      int warps_per_cta, int region_bytes, cudaStream_t stream);
cudaError_t sd_occupancy(bool sparse, bool smem, bool flat, int warps_per_cta, int region_bytes,
                         int table_bytes, int *ctas_per_sm);
// Rotor kernel; `stage` is its state location (kStageShared only for the
// proposals that keep delta energies, 0 and 1).
cudaError_t launch_rmc(bool random_order, int proposal, int stage, const RmcArgs &args, int grid,
                       int warps_per_cta, cudaStream_t stream);
// One thread per sample (proposals 2 and 3).
cudaError_t launch_rmc_thread(bool random_order, int proposal, const RmcArgs &args,
                              cudaStream_t stream);
cudaError_t rmc_occupancy(bool random_order, int proposal, int stage, int warps_per_cta,
                          int64_t region_bytes, int *ctas_per_sm);
cudaError_t launch_pimc(bool chain_update, const PimcArgs &args, int grid, int block,
                        cudaStream_t stream);
// Single-qubit updates, one warp per sample.
cudaError_t launch_pimc_warp(const PimcArgs &args, int grid, int warps_per_cta, int warp_bytes,
                             cudaStream_t stream);
cudaError_t acceptance_check(int64_t samples, uint64_t seed, unsigned long long *d_counts);
cudaError_t bounds_check(int64_t samples, uint64_t seed, unsigned long long *d_counts);

}  // namespace b200sa
