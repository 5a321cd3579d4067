// Types shared by the host packer, the launch code and the sm_100a kernels.
#pragma once
#include <cmath>
#include <cstdint>

#include <vector_types.h>

#ifndef __CUDACC__
#define __host__
#define __device__
#endif

namespace b200sa {

// RNG output ring per read (shared memory).  The ring holds the next
// kRing outputs of the read's xorshift128+ stream; it is refilled one half at
// a time, each lane producing kPerLane consecutive outputs from its own
// segment-start state, and each lane then jumps that state kHalf steps ahead
// with a precomputed GF(2) matrix (xorshift128+ is linear over GF(2)).
constexpr int kRing = 256;
constexpr int kHalf = kRing / 2;
constexpr int kPerLane = kHalf / 32;

// Per-variable adjacency record (uint2): x = start of the variable's list,
// y = its degree (list length).
constexpr uint32_t kDegMask = 0x00ffffffu;
constexpr uint32_t kMaxDegree = kDegMask;

// Speculation arrays, read once per variable and pass (kept as two compact
// arrays, 5 bytes per variable, so they stay in the L1 left beside the
// shared regions):
//   dist:  distance to the nearest later neighbour (u - v for the smallest
//          neighbour u > v), capped at kDistCap.  A flip of v can only change
//          the decision of a later variable of the current window if that
//          variable is at least this far ahead.
//   share: conflict mask.  Bit 0 is set when v's list names a target twice;
//          bit j (1..31) when v and v + j have a common neighbour.  Two
//          committed flips can add into the same delta-energy slot only
//          through one of these.
constexpr uint32_t kDistCap = 32;  // the speculative window

struct ProblemDev {
    int32_t n;
    int32_t sweeps_per_beta;
    int32_t num_betas;
    int32_t num_reads;
    int64_t m;              // couplers
    int64_t state_offset;   // element offset of read 0 in the state arrays
    int64_t read_offset;    // offset of read 0 in energies / seeds / stats
    const uint2 *vinfo;     // [n] adjacency record (see above)
    const uint8_t *dist;    // [n] speculation distance (see above)
    const uint32_t *share;  // [n] conflict mask (see above)
    const int32_t *col;     // [2m] neighbour index, coupler input order
    const double *w;        // [2m] coupling
    const double *h;        // [n]
    const int32_t *cu;      // [m] COO, input order (energy)
    const int32_t *cv;      // [m]
    const double *cw;       // [m]
    const double *betas;    // [num_betas]
    const double *thresholds;  // [num_betas] 44.36142 / beta, host-divided
    int32_t varorder;       // 0 sequential, 1 random
    int32_t proposal;       // 0 Gibbs, 1 Metropolis
    // Every adjacency list has this length (1..32) and list v starts at
    // v * regular_degree; 0 when the lists differ in length.
    int32_t regular_degree;
    uint32_t regular_magic;  // ceil(2^16 / regular_degree): t / D == (t * magic) >> 16 for t < 1024
    // In-window resolution of the sequential sweep (1: on, for reads whose
    // spins are all +-1).  back[v] = {mask, start}: bit o (1..31) of mask set
    // when v - o is a neighbour of v; bw[start ..] the couplings of those
    // neighbours, offsets descending (the order the reference adds their
    // flips' contributions).  No list may name a target twice.
    int32_t resolve;
    // State in registers (sa_dense.cuh; 1: on): a coupling matrix, row j of
    // dense_w holding the couplings of variable j (0 where there is none), rows
    // padded to a multiple of 32, kDenseMaxN readable entries after the last row.
    // n <= kDenseMaxN, no list names a target twice.
    int32_t dense;
    const uint2 *back;
    const double *bw;
    // The conflict mask (share) of windows of 32 variables from a multiple of 32
    // on, without entries naming a later variable of the same window.
    const uint32_t *wshare;
    const double *dense_w;
    // Banded delta energies (kStageBand): adjacency entries mostly within
    // band_b of their variable; band_w is the shared-memory ring size (a power
    // of two >= 2 band_b + 128), 0 when the problem is not banded.
    int32_t band_b;
    int32_t band_w;
};
constexpr int kDenseSlots = 10;  // variables per lane at most
constexpr int kDenseMaxN = 32 * kDenseSlots;
__host__ __device__ inline int dense_ld(int n) { return (n + 31) & ~31; }
constexpr int kBandMaxSlots = 8192;  // 64 KB of delta energies per warp at most
// Equal lists up to this length are staged beside the band, two windows of
// them (12 bytes an entry).
constexpr int kListMaxDegree = 8;
constexpr int kListBytes = 2 * 32 * kListMaxDegree * 12;

// Per-read counters written by the kernel.
struct ReadStats {
    unsigned long long flips;
    unsigned long long passes;
    unsigned int near_ties;
    unsigned int pad;
};

struct LaunchArgs {
    const ProblemDev *problems;
    const int64_t *items;          // (problem << 32) | read, execution order
    int64_t num_items;
    unsigned long long *queue_head;  // persistent mode work-queue head (nullptr: static)
    const int8_t *states_in;
    int8_t *states_out;
    double *energies;
    const uint64_t *seeds;         // indexed by read_offset + r
    ReadStats *stats;              // indexed by read_offset + r
    int32_t shared_stream;         // 1: one warp, items in order, one RNG stream
    uint64_t *rng_carry;           // shared-stream state between launches
    int32_t carry_in;              // 1: resume the stream from rng_carry
    int32_t smem_cap_n;            // largest n kept in the warp's shared region
    double *scratch_de;            // global fallback state, one slot per warp
    int8_t *scratch_s;
    int64_t scratch_stride;        // elements per slot
    int64_t num_slots;
    // Random order: bytes of the per-warp bitmap of variables touched by the
    // window's accepted flips (touch_bytes_for of the launch's largest n), in
    // the shared region between the scratch and the state; 0 otherwise.
    int32_t touch_bytes;
    // kStageBand: slots of the per-warp delta-energy band (0 otherwise).
    int32_t band_cap;
};

// Arguments of the steepest-descent kernel (sd_kernel.cuh): one problem,
// items (0 << 32) | sample taken from a queue head.
struct SdArgs {
    const ProblemDev *problem;
    const int64_t *items;        // (0 << 32) | sample
    int64_t num_items;
    unsigned long long *queue_head;
    const int8_t *states_in;
    int8_t *states_out;
    double *energies;
    uint32_t *steps;
    uint32_t max_steps;
    double *scratch_fe;          // per-warp global slots, or null: state in shared memory
    int8_t *scratch_s;
    int64_t scratch_stride;
    int32_t table_bytes;         // list starts at the head of a CTA's shared memory
    int32_t any_dup;             // some list names a target twice
    unsigned long long *scratch_key;  // group minima (sd_kernel.cuh)
    uint8_t *scratch_at;
    int64_t group_stride;
    unsigned long long *capped;  // samples stopped by max_steps
};

// Per-warp shared region of the descent kernel: 32 doubles for equal-target
// sums, then (state in shared memory) flip energies, group keys, spins and the
// places of the group minima.
constexpr int kSdScratchBytes = 32 * 8;  // equal-target sums
// List starts, one table per CTA (state in shared memory, lists of different
// lengths).
inline int64_t sd_table_bytes(int64_t n) { return (4 * (n + 1) + 15) & ~int64_t(15); }
inline int64_t sd_region_bytes(int64_t cap_n) {
    const int64_t groups = (cap_n + 31) / 32;
    return (kSdScratchBytes + 8 * (cap_n + groups) + cap_n + groups + 15) & ~int64_t(15);
}

// Whether a step looks at every variable instead of the group minima: with few
// groups, and where a flip's list is long enough to change most of them (mean
// degree n / 12 and more).  Group minima against all variables, whole calls of
// 8192 samples (ms): n = 128 degree 6 0.93, 0.91; n = 300 degree 3 1.30, 1.32,
// degree 50 2.64, 2.45, complete 12.0, 11.0; n = 500 degree 25 2.69, 2.78, degree
// 50 4.08, 3.86; n = 1000 degree 50 7.98, 8.42, degree 100 14.1, 13.5; n = 2048
// degree 6 7.7, 13.0, degree 100 33.3, 33.2, degree 200 62.3, 56.4.
inline bool sd_flat(int64_t n, int64_t m) { return n <= 256 || 24 * m >= n * n; }

// Arguments of the rotor-model annealing kernel (rmc_kernel.cuh).
struct RmcArgs {
    int32_t n;
    int64_t m;
    const uint2 *vinfo;      // [n] {list start, degree}
    const int32_t *col;      // adjacency, coupler input order
    const double *w;
    const double *h;
    const double *tf;        // [n] transverse fields
    const int32_t *cu, *cv;  // COO (energy order)
    const double *cw;
    const double *hp, *hd;   // [num_betas] problem and driver field schedules
    int32_t num_betas;
    int32_t sweeps_per_beta;
    const uint64_t *seeds;
    int32_t shared_stream;   // 1: one warp, samples in order, one RNG stream
    int32_t num_samples;
    uint8_t *rows;           // [num_samples][n] initial states in, final states out
    const uint8_t *dist;     // [n] speculation distance (ProblemDev::dist)
    const uint32_t *share;   // [n] conflict mask (ProblemDev::share)
    int32_t regular_degree;  // ProblemDev::regular_degree, regular_magic
    uint32_t regular_magic;
    int32_t region_bytes;    // a warp's shared region (rmc_region_bytes)
    int32_t touch_bytes;     // random order: bytes of a warp's touch bitmap
    uint32_t *touch;         // the bitmaps, one per warp, or null: in the region
    double *de;              // per-warp global slots of slot_stride elements
    uint8_t *states;         // (state locations kStageSpins and kStageGlobal);
    int64_t slot_stride;     // one thread per sample: both [n][num_samples]
    double *energies;
    uint8_t *stats;          // [num_samples][points][n], or null
    int32_t interval;
    const double *cos_table, *sin_table;  // [256]
    unsigned long long *near;
};

// Shared memory of the rotor kernel: the two angle tables per CTA, then per
// warp the RNG ring, scratch, touch bitmap and, by the state location, delta
// energies (proposals that keep them) and angles.
constexpr int kRmcTableBytes = 2 * 256 * 8;
constexpr int kRmcMaxWarps = 8;  // warps per CTA
// Above this many samples rotor annealing runs one thread per sample (all
// proposals; per-sample streams).  A thread's time per attempt hardly grows until
// the samples fill the chip, a warp's grows with the samples from about 12 warps
// per SM on, and a warp's windows are mostly empty when there are few variables.
// Both sides measured as whole calls, 1000 attempts a sample, degree 4 (ms, warp
// against thread), n from 5 to 1024 and 1024 to 262144 samples, and degrees 3, 8
// and 20; the line lies where they meet or a little to the warp's side:
//   reflections, sequential  n = 16: 4096 samples 0.88, 0.82; n = 32: 8192 1.07,
//     0.90; n = 128: 16384 1.49, 1.60, 65536 4.9, 3.3; n = 256: 65536 6.4, 6.4
//   reflections, random      n = 32: 2048 1.20, 1.32, 4096 2.1, 1.35; n = 64: 4096
//     1.54, 1.37; n = 128: 16384 3.0, 3.8, 65536 10.0, 6.4; n = 256: 65536 10.4, 11.9
//   angles, sequential       n = 32: 4096 1.06, 1.08; n = 256: 8192 1.60, 1.62; n =
//     1024: 16384 8.4, 8.1
//   angles, random           n = 32: 2048 1.45, 1.53; n = 64: 4096 1.88, 1.56; n =
//     256: 8192 2.26, 2.05; n = 512: 16384 6.7, 9.3, 32768 12.2, 11.1
// Beyond 128 variables a thread's delta energies leave the caches.
inline int64_t rmc_thread_samples(int proposal, bool random_order, int n) {
    const int64_t never = INT32_MAX;
    if (proposal <= 1) {
        if (n > 128) return never;
        if (!random_order) return n <= 16 ? 4096 : 256 * (int64_t)n;
        return n <= 32 ? 2560 : n <= 64 ? 80 * (int64_t)n : 32768;
    }
    if (!random_order) return 4096 + 16 * (int64_t)n;
    return n <= 53 ? 2560 : n <= 256 ? 48 * (int64_t)n : 64 * (int64_t)n;
}

// Arguments of the path-integral Monte Carlo kernels (pimc_kernel.cuh): a warp
// per sample, mt19937 state and scratch in shared memory, or a thread per sample
// (a "slot"), both in global memory.  Break lists have a fixed capacity per
// variable; proposals and domains per update have one too.
struct PimcArgs {
    int32_t n;
    int64_t m;
    const uint2 *vinfo;      // [n] {list start, degree}
    const int32_t *col;      // adjacency, coupler input order
    const double *w;
    const double *h;
    const int32_t *cu, *cv;  // COO (energy order)
    const double *cw;
    const double *hp, *hd;   // [num_betas] problem (invTemp) and driver (Gamma) schedules
    int32_t num_betas;
    int32_t sweeps_per_beta;
    double jchain;           // chain coupling (Swendsen-Wang joins)
    int32_t qpc;             // qubits per chain (chain update)
    int32_t chains;          // n / qpc
    const uint32_t *seeds;
    int32_t shared_stream;   // 1: one warp or thread, samples in order, one generator
    int32_t num_samples;
    int8_t *states;          // [num_samples][n], the first Trotter slice
    int32_t *counts;         // [num_samples][n] breaks per variable
    int32_t *breaks;         // [num_samples][n][list_stride]
    int32_t cap_breaks;
    int32_t list_stride;     // cap_breaks, rounded up to 16 bytes
    int32_t cap_props;       // proposals per qubit and update
    uint32_t *mt;            // [slots][kMtWords]; null (as the scratch) for a warp per sample
    int32_t *scratch_i;      // [slots][scratch_ints]
    double *scratch_d;       // [slots][scratch_doubles]
    int64_t scratch_ints, scratch_doubles;
    double *energies;
    int8_t *stats;           // [num_samples][points][n], or null
    int32_t interval;
    unsigned long long *near;
    int32_t *overflow;       // set when a capacity would be exceeded
};
constexpr int kMtWords = 624;
constexpr int kPimcSlices = 65536;  // numTrotterSlices, localPIMC.h:88
// Warps per CTA of the warp-per-sample kernel at most, and its shared memory
// per sample: mt19937 state, scratch (PimcWarpScratch).
constexpr int kPimcMaxWarps = 4;
// Above this many samples single-qubit updates run one thread per sample.  A
// warp's update costs nearly the same whatever it finds; a thread's grows with
// the domains (the transverse field, here its mean over the schedule), with the
// neighbours and with the distance of its lists, and hardly with the samples
// until they fill the chip.  Where the two meet, as whole calls of a field
// falling geometrically to 0.05 (mean 0.14, 0.32 and 1.07; samples): n = 5:
// 9000, 12500, 22500; n = 12 degree 4 12000, 16000, 36000, degree 11 14500, 18000,
// 41000; n = 32 degree 4 14500, 19500, 42000, degree 12 20000, 28000, 62000; n =
// 128 degree 4 18500, 33000, beyond, degree 12 33500, 50000, beyond; n = 512
// degree 4 22500.  The product below follows these; from n = 512 on the samples'
// lists leave the caches and the line lies near 42000 (degree 6, field 5 ->
// 0.05, 16 steps, kernel time of a warp and of a thread: 16384 samples 151, 249
// ms, 32768 288, 315, 65536 566, 497), so it ends there.
inline int64_t pimc_thread_samples(int64_t n, int64_t m, double mean_field) {
    const double degree = 2.0 * (double)m / (double)n;
    const double line = 4350.0 * (1.0 + 2.65 * mean_field) * (1.0 + degree / 12.0) *
                        std::pow((double)n, 1.0 / 6.0);
    return line < 40960.0 ? (int64_t)line : 40960;
}
inline int64_t pimc_warp_bytes(int64_t cap_props, int64_t cap_breaks) {
    const int64_t cap = cap_props + cap_breaks;
    return (4 * kMtWords + 32 * (8 + 4 + 4) + 8 * cap + cap + 15) & ~int64_t(15);
}

// Nibble tables of the RNG jump matrix: entry [k][v] is the jump applied to
// the state whose only set bits are the nibble value v at nibble position k.
constexpr int kJumpNibbles = 32;
constexpr int kJumpTable = kJumpNibbles * 16;

// Shared-stream carry layout (uint64 words).
constexpr int kCarryLaneWords = 64;                 // 32 lanes x 2 words
constexpr int kCarryWords = kRing + kCarryLaneWords + 2;  // ring, lanes, q, base

// Per-warp shared region: RNG ring, scratch (32 doubles for equal-slot sums,
// 32 ints for the rank table of accepted flips; then the lanes' RNG
// segment-start states and the read's counters, which the sweep loop keeps
// out of registers), delta energies, spins.  (region_bytes_for keeps every
// region a multiple of 16 bytes.)
constexpr int kScratchHotBytes = 32 * 8 + 32 * 4;
constexpr int kColdBytes = 32 * 16 + 32;
constexpr int kScratchBytes = kScratchHotBytes + kColdBytes;
inline int region_bytes_for(int cap_n) {
    const int spins = (cap_n + 15) & ~15;
    return kRing * 8 + kScratchBytes + ((cap_n * 8 + 15) & ~15) + spins;
}

// Where a read's state lives: kStageGlobal keeps delta energies and spins in
// a per-warp global slot (L2-resident), kStageShared both in the warp's
// shared region, kStageSpins the spins in the shared region and the delta
// energies in the global slot (a smaller global footprint, and the spin
// reads of the neighbour updates stay on chip).
constexpr int kStageGlobal = 0;
constexpr int kStageShared = 1;
constexpr int kStageSpins = 2;
// kStageBand: spins in the shared region, the delta energies of a band of
// variables around the window in a shared-memory ring after them (band_cap
// slots), the others in the global slot (sequential order, banded problems).
constexpr int kStageBand = 3;
constexpr int kNumStages = 4;
inline int region_bytes_for_stage(int stage, int cap_n, int band_cap = 0) {
    if (stage == kStageShared) return region_bytes_for(cap_n);
    if (stage == kStageSpins) return kRing * 8 + kScratchBytes + ((cap_n + 15) & ~15);
    if (stage == kStageBand) return kRing * 8 + kScratchBytes + ((cap_n + 15) & ~15) + 8 * band_cap + kListBytes;
    return kRing * 8 + kScratchBytes;
}

// Rotor kernel: kStageShared delta energies and angles, kStageSpins angles,
// kStageGlobal neither.
inline int64_t rmc_region_bytes(int stage, int64_t n, int touch_bytes) {
    const int64_t angles = (n + 15) & ~int64_t(15);
    return kRing * 8 + kScratchBytes + touch_bytes + (stage != kStageGlobal ? angles : 0) +
           (stage == kStageShared ? (n * 8 + 15) & ~int64_t(15) : 0);
}

// Random order keeps a bitmap of n bits per warp (16-byte multiple).
inline int touch_bytes_for(bool random_order, int max_n) {
    return random_order ? (((max_n + 31) / 32) * 4 + 15) & ~15 : 0;
}

}  // namespace b200sa
