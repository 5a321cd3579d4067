// Simulated-annealing sweep for sm_100a: one warp per read.
//
// Arithmetic follows dwave-samplers 1.8.0 dwave/samplers/sa/src/cpu_sa.cpp
// operation for operation (explicit __dadd_rn/__dmul_rn, so no contraction
// can change a rounding):
//   local field / initial delta energy   cpu_sa.cpp:54-74, 113-116
//   skip threshold 44.36142/beta          cpu_sa.cpp:131, 140 (host-divided)
//   Metropolis / Gibbs acceptance         cpu_sa.cpp:144-166
//   neighbour delta-energy update         cpu_sa.cpp:172-190
//   state energy                          cpu_sa.cpp:210-227
//   xorshift128+                          cpu_sa.cpp:27-34, seeding :283-284
//
// Sequential order runs in speculative passes over a window of up to 32
// consecutive variables (one per lane).  Every lane evaluates its decision
// against the delta energies as they stand at the start of the pass; the RNG
// draw each lane would consume is placed by a prefix count of the lanes
// before it that need a draw.  A flip of variable v invalidates only lanes at
// or beyond v + dist(v), dist being the distance to v's nearest later
// neighbour, so the pass commits the prefix of lanes before the smallest such
// bound.  The committed prefix is exactly what the reference computes
// one variable at a time: its delta energies were untouched by earlier flips
// in the window and its draws land on the same stream positions.
//
// Committed flips are pairwise non-adjacent, so their neighbour updates never
// touch each other's slots or spins.  They are applied together: the
// adjacency entries of all committed flips, concatenated in variable order,
// are spread over the lanes 32 at a time.  Entries that name the same slot
// (a neighbour shared by two flips, or a self-loop / repeated coupler) are
// grouped with __match_any_sync and added by the group's first lane in entry
// order, so every slot receives its additions in the reference's order.  The
// grouping is skipped when the per-variable conflict masks (computed at pack
// time) show that no two entries of the pass can name the same slot.  Slots in
// global memory receive their additions as L2 reductions (see GlobalDe).
#pragma once
#include <cstdint>

#include "sa_types.h"

namespace b200sa {

// Nibble tables of the GF(2) matrix (xorshift128+ transition)^kHalf.
__device__ uint4 g_jump_nib[kJumpTable];

constexpr unsigned kFull = 0xffffffffu;
constexpr double kTwo64 = 18446744073709551616.0;  // (double)RANDMAX
// Width of the band around an exp() decision inside which CUDA's exp and
// the host libm's exp (each within ~1 ulp of the true value) could disagree.
constexpr double kTieRel = 3.552713678800501e-15;  // 2^-48

// Stream positions are kept modulo 2^32: only their differences (all below
// kRing) and their residues modulo kRing are used, and both survive the wrap.
struct RingState {
    uint32_t q;     // outputs consumed so far (stream position, warp-uniform)
    uint32_t base;  // ring holds positions [base, base + kRing)
};

// Per-warp words the sweep loop touches rarely, kept in the warp's shared
// region after the conflict scratch (kColdBytes): each lane's segment-start
// state for the next ring refill (once per kHalf draws) and the read's
// counters (added to by lane 0 once per sweep).  Every member is accessed
// with 8-byte (or smaller) loads and stores, so the region needs only the
// 8-byte alignment of the ring before it.
struct WarpCold {
    uint64_t seg[64];  // lane l: words 2l, 2l + 1
    unsigned long long flips;
    unsigned long long passes;
    unsigned int near;
    unsigned int pad[3];
};
static_assert(sizeof(WarpCold) == kColdBytes, "cold words");

// The ring is followed by the scratch (kScratchHotBytes), then WarpCold.
__device__ __forceinline__ WarpCold *warp_cold(uint64_t *ring) {
    return reinterpret_cast<WarpCold *>(reinterpret_cast<uint8_t *>(ring + kRing) +
                                        kScratchHotBytes);
}

// One sweep's counts (warp-uniform; at most n each), added by lane 0 to the
// read's counters when the sweep ends.
struct SweepCount {
    unsigned flips = 0, passes = 0, near = 0;
    __device__ __forceinline__ void pass(unsigned f, unsigned nt) {
        flips += f;
        passes += 1;
        near += nt;
    }
    __device__ __forceinline__ void flush(uint64_t *ring, unsigned lane) const {
        if (lane == 0) {
            WarpCold *c = warp_cold(ring);
            c->flips += flips;
            c->passes += passes;
            c->near += near;
        }
    }
};

// ---- acceptance tests ------------------------------------------------------
// The reference decides Metropolis as exp(x) * 2^64 > (double)rand with
// x = -dE*beta (cpu_sa.cpp:154) and Gibbs as 2^64 > (double)rand * (1 +
// exp(z)) with z = dE*beta (cpu_sa.cpp:163).  Both are first decided in the
// log2 domain with single-precision hardware approximations, whose total
// error is below 2^-14 in log2 units for the argument ranges that reach them
// (|x| < 44.4 and z < 44.4 since dE < 44.36142/beta): every term's error is
// bounded by a few single-precision roundings of magnitudes <= 110 plus the
// lg2/ex2 approximation error (relative 2^-22).  When the two sides differ by
// more than kBand = 2^-10 the fast answer equals the exact one; otherwise the
// exact double-precision expression is evaluated.  The band is reached by
// about 0.1% of draws.
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kBand = 0.0009765625f;  // 2^-10

__device__ __forceinline__ float lg2_approx(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float ex2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1 accept, 0 reject, -1 undecided.  x = -dE*beta in (-44.4, 0].
__device__ __forceinline__ int metropolis_fast(double x, uint64_t r) {
    const float t = __fmaf_rn((float)x, kLog2e, 64.0f);  // log2(exp(x) * 2^64)
    const float y = lg2_approx(__ull2float_rn(r));      // log2(rand); -inf at 0
    if (t > y + kBand) return 1;
    if (t < y - kBand) return 0;
    return -1;
}

// 1 accept, 0 reject, -1 undecided.  z = dE*beta < 44.4 (may be -inf).
__device__ __forceinline__ int gibbs_fast(double z, uint64_t r) {
    const float zf = (float)z;
    float g;  // log2(1 + exp(z))
    if (zf > 24.0f)
        g = zf * kLog2e;  // log2(1 + exp(-z)) < 2^-33 omitted
    else if (zf < -24.0f)
        g = 0.0f;  // log2(1 + exp(z)) < 2^-33
    else
        g = lg2_approx(1.0f + ex2_approx(zf * kLog2e));
    const float s = lg2_approx(__ull2float_rn(r)) + g;  // log2(rand * (1 + exp(z)))
    if (s < 64.0f - kBand) return 1;
    if (s > 64.0f + kBand) return 0;
    return -1;
}

// The exact double-precision decisions, reached only inside the band.  Kept
// out of line so the sweep loop does not hold exp()'s registers.
// Returns accept in bit 0 and the near-tie flag in bit 1.
__device__ __noinline__ int metropolis_exact(double d, double beta, uint64_t r) {
    const double rd = __ull2double_rn(r);
    const double e = exp(__dmul_rn(-d, beta));  // cpu_sa.cpp:152-154
    const double x = __dmul_rn(e, kTwo64);
    return (x > rd ? 1 : 0) | (fabs(x - rd) <= x * kTieRel ? 2 : 0);
}

__device__ __noinline__ int gibbs_exact(double d, double beta, uint64_t r) {
    const double rd = __ull2double_rn(r);
    const double e = exp(__dmul_rn(d, beta));  // cpu_sa.cpp:162-163
    const double y = __dmul_rn(rd, __dadd_rn(1.0, e));
    return (kTwo64 > y ? 1 : 0) | (fabs(y - kTwo64) <= kTwo64 * kTieRel ? 2 : 0);
}

// A field of the problem record read again at each use, for values used once
// per sweep that are not worth a register through the sweep loop.  The load
// goes through the read-only cache (ld.global.nc, an L1 hit after the first
// sweep); the asm statement is volatile so that the compiler does not hoist
// it out of the loop.  The record does not change while a kernel runs.
__device__ __forceinline__ int reload(const int &x) {
    int r;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(r) : "l"(&x));
    return r;
}
template <class T>
__device__ __forceinline__ T *reload(T *const &x) {
    unsigned long long r;
    asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(r) : "l"(&x));
    return reinterpret_cast<T *>(r);
}

// Problem fields the sweep loop keeps in registers (fields used only when a
// read starts or ends are read from the ProblemDev record there).
struct Prob {
    int n;
    const ProblemDev *pd;  // the schedule is read from here once per beta
    const uint2 *__restrict__ vinfo;
    const int32_t *__restrict__ col;
    const double *__restrict__ w;
    const uint8_t *__restrict__ dist;
    const uint32_t *__restrict__ share;
    const uint32_t *__restrict__ wshare;
    int regular_degree;
    uint32_t regular_magic;
    const uint2 *__restrict__ back;
    const double *__restrict__ bw;
};

__device__ __forceinline__ Prob load_prob(const ProblemDev *P) {
    Prob q;
    q.n = P->n;
    q.pd = P;
    q.vinfo = P->vinfo;
    q.col = P->col;
    q.w = P->w;
    q.dist = P->dist;
    q.share = P->share;
    q.wshare = P->wshare;
    q.regular_degree = P->regular_degree;
    q.regular_magic = P->regular_magic;
    q.back = P->back;
    q.bw = P->bw;
    return q;
}

// Brings the line holding *p (global memory) into L1 without waiting.
__device__ __forceinline__ void prefetch_l1(const void *p) {
    asm volatile("prefetch.global.L1 [%0];" : : "l"(p));
}

// Accessors of a read's delta energies, one per state location: get, set and
// add (de[x] = de[x] + v, rounded to nearest like the reference's `+=`,
// cpu_sa.cpp:172-185).  kAsyncAdd: an add does not wait for memory.
//
// SharedDe: the warp's shared region (kStageShared).
struct SharedDe {
    static constexpr bool kAsyncAdd = false;
    double *p;
    __device__ __forceinline__ double get(int x) const { return p[x]; }
    __device__ __forceinline__ void set(int x, double v) const { p[x] = v; }
    __device__ __forceinline__ void add(int x, double v) const { p[x] = __dadd_rn(p[x], v); }
};

// GlobalDe: the warp's global slot (kStageGlobal, kStageSpins), L2-resident.
// An add is a reduction performed at L2 (red.global.add.f64, round to
// nearest even, the same rounding as a load, __dadd_rn and a store), so the
// update phase issues its additions without waiting for the slots' values.
// Two adds to one slot from one thread land in program order, and a barrier
// of the warp orders them before any later access by its lanes.  Reads go to
// L2 (ld.global.cg), where the reductions are performed, never to a line an
// earlier read left in L1.
struct GlobalDe {
    static constexpr bool kAsyncAdd = true;
    double *p;
    __device__ __forceinline__ double get(int x) const { return __ldcg(p + x); }
    __device__ __forceinline__ void set(int x, double v) const { __stcg(p + x, v); }
    __device__ __forceinline__ void add(int x, double v) const {
        asm volatile("red.global.add.f64 [%0], %1;" : : "l"(p + x), "d"(v) : "memory");
    }
};

// BandDe: a banded problem (kStageBand).  The slots of the variables in
// [lo, lo + w) live in a shared-memory ring (`b`, w a power of two, slot
// x & (w - 1)); every other variable's slot is in the global array `g`.  The
// band slides with the window (see sweep_sequential) and fetches its slots
// with cp.async through L1, so the global part is read and written with plain
// loads and stores.  With w = 0 everything is global.
struct BandDe {
    static constexpr bool kAsyncAdd = false;
    double *g;
    double *b;
    int lo;
    unsigned w;
    __device__ __forceinline__ double &at(int x) const {
        return (unsigned)(x - lo) < w ? b[(unsigned)x & (w - 1u)] : g[x];
    }
    __device__ __forceinline__ double get(int x) const { return at(x); }
    __device__ __forceinline__ void set(int x, double v) const { at(x) = v; }
    __device__ __forceinline__ void add(int x, double v) const {
        double &s = at(x);
        s = __dadd_rn(s, v);
    }
};

template <int STAGE>
struct DeFor {
    using T = GlobalDe;
};
template <>
struct DeFor<kStageShared> {
    using T = SharedDe;
};
template <>
struct DeFor<kStageBand> {
    using T = BandDe;
};

// 8-byte asynchronous copy global -> shared (completes at cp_async_wait).
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" : : "r"(s), "l"(gmem) : "memory");
}
// The same for 16 bytes, both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" : : "r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" : : : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" : : "n"(N) : "memory");
}

__device__ __forceinline__ void xs_advance(uint64_t &s0, uint64_t &s1) {
    uint64_t a = s0;
    const uint64_t b = s1;
    s0 = b;
    a ^= a << 23;
    s1 = a ^ b ^ (a >> 17) ^ (b >> 26);
}

__device__ __forceinline__ uint64_t xs_next(uint64_t &s0, uint64_t &s1) {
    const uint64_t b = s1;
    xs_advance(s0, s1);
    return s1 + b;
}

// State <- M * state over GF(2), M = (xorshift128+ transition)^kHalf: the
// XOR of one table entry per nibble of the 128-bit state (32 lookups).
__device__ __forceinline__ void xs_jump(uint64_t &s0, uint64_t &s1) {
    uint32_t a0 = 0, a1 = 0, a2 = 0, a3 = 0;
#pragma unroll
    for (int k = 0; k < kJumpNibbles; ++k) {
        const uint64_t word = k < 16 ? s0 : s1;
        const uint32_t nib = (uint32_t)(word >> (4 * (k & 15))) & 15u;
        const uint4 c = __ldg(&g_jump_nib[k * 16 + nib]);
        a0 ^= c.x;
        a1 ^= c.y;
        a2 ^= c.z;
        a3 ^= c.w;
    }
    s0 = (uint64_t)a0 | ((uint64_t)a1 << 32);
    s1 = (uint64_t)a2 | ((uint64_t)a3 << 32);
}

// Lane l writes stream positions pos + l*kPerLane + t, t < kPerLane, starting
// from the state that precedes position pos + l*kPerLane.
__device__ __forceinline__ void ring_fill(uint64_t *ring, uint32_t pos,
                                          uint64_t s0, uint64_t s1,
                                          unsigned lane) {
    const uint32_t start = pos + lane * (uint32_t)kPerLane;
#pragma unroll
    for (int t = 0; t < kPerLane; ++t)
        ring[(start + t) & (kRing - 1)] = xs_next(s0, s1);
}

__device__ __forceinline__ void ring_init(uint64_t *ring, RingState &rs,
                                          uint64_t seed, unsigned lane) {
    uint64_t s0 = seed ? seed : ~0ull, s1 = 0;  // cpu_sa.cpp:283-284
    for (unsigned k = 0; k < lane * kPerLane; ++k) xs_advance(s0, s1);
    __syncwarp();
    ring_fill(ring, 0, s0, s1, lane);
    xs_jump(s0, s1);
    ring_fill(ring, kHalf, s0, s1, lane);
    xs_jump(s0, s1);
    uint64_t *seg = warp_cold(ring)->seg + 2 * lane;
    seg[0] = s0;
    seg[1] = s1;
    rs.q = 0;
    rs.base = 0;
    __syncwarp();
}

// Overwrites the consumed lower half with the positions kRing further on and
// advances this lane's segment-start state.  Out of line: it runs once per
// kHalf draws.
__device__ __noinline__ void ring_refill_half(uint64_t *ring, uint32_t pos, unsigned lane) {
    __syncwarp();
    uint64_t *seg = warp_cold(ring)->seg + 2 * lane;
    uint64_t s0 = seg[0], s1 = seg[1];
    ring_fill(ring, pos, s0, s1, lane);
    xs_jump(s0, s1);
    seg[0] = s0;
    seg[1] = s1;
    __syncwarp();
}

// Keeps positions [q, q + kHalf) available: once the lower half is consumed
// it is overwritten with the positions kRing further on.
__device__ __forceinline__ void ring_refill(uint64_t *ring, RingState &rs,
                                            unsigned lane) {
    if (rs.q - rs.base >= (uint32_t)kHalf) {
        ring_refill_half(ring, rs.base + kRing, lane);
        rs.base += kHalf;
    }
}

// cpu_sa.cpp:54-74 for every variable, then the working copy of the spins.
// Returns (warp-uniform) whether every spin is +1 or -1.
__device__ __forceinline__ bool load_state(const ProblemDev *PD, const int8_t *src,
                                           double *de, int8_t *sp,
                                           unsigned lane) {
    const int n = PD->n;
    const uint2 *__restrict__ vinfo = PD->vinfo;
    const int32_t *__restrict__ col = PD->col;
    const double *__restrict__ w = PD->w;
    const double *__restrict__ h = PD->h;
    bool pm1 = true;
    for (int v = lane; v < n; v += 32) {
        const int8_t x = src[v];
        sp[v] = x;
        pm1 = pm1 && (x == 1 || x == -1);
    }
    pm1 = __all_sync(kFull, pm1);
    __syncwarp();
    for (int v = lane; v < n; v += 32) {
        const uint2 vi = __ldg(&vinfo[v]);
        const int e1 = (int)vi.x + (int)(vi.y & kDegMask);
        double f = __ldg(&h[v]);
#pragma unroll 4
        for (int e = (int)vi.x; e < e1; ++e)
            f = __dadd_rn(f, __dmul_rn((double)(int)sp[__ldg(&col[e])], __ldg(&w[e])));
        de[v] = __dmul_rn((double)(-2 * (int)sp[v]), f);
    }
    __syncwarp();
    return pm1;
}

// The additions of entries `grp` (lanes, in entry order; values in
// scratch) to one slot, in that order.
template <class DE>
__device__ __forceinline__ void add_group(const DE &de, int x, unsigned grp, const double *scratch) {
    if constexpr (DE::kAsyncAdd) {
        while (grp) {
            const int j = __ffs(grp) - 1;
            grp &= grp - 1;
            de.add(x, scratch[j]);
        }
    } else {
        double acc = de.get(x);
        while (grp) {
            const int j = __ffs(grp) - 1;
            grp &= grp - 1;
            acc = __dadd_rn(acc, scratch[j]);
        }
        de.set(x, acc);
    }
}

// The flips of `rest` without an earlier flip in it that shares a neighbour
// (`shr` is the lane's conflict mask, ProblemDev::share): applied together they
// name no slot twice, and applied before the others they keep the order of
// additions.
__device__ __forceinline__ unsigned first_phase(unsigned rest, uint32_t shr, unsigned lane) {
    unsigned partners = 0u;
    if (lane < 31 && ((rest >> lane) & 1u))
        partners = ((shr >> 1) & (rest >> (lane + 1))) << (lane + 1);
    return rest & ~__reduce_or_sync(kFull, partners);
}

// Adds x[i] to slot nb[i] (none when negative) of N entries per lane, entry i
// belonging to the flip of lane k[i], in phases (first_phase) with a barrier
// between two of them, so additions to one slot from different lanes land in
// the order of the phases.  What is left after kPhases of them (hubs that most
// flips share) is matched, 32 entries at a time.
constexpr int kPhases = 3;
template <int N, class DE>
__device__ __forceinline__ void add_phased(const DE &de, const int (&nb)[N], const double (&x)[N],
                                           const int (&k)[N], unsigned fm, uint32_t shr,
                                           double *scratch, unsigned lane) {
    unsigned rest = fm;
    for (int phase = 0; phase < kPhases && rest; ++phase) {
        const unsigned now = first_phase(rest, shr, lane);
        bool on[N];
#pragma unroll
        for (int i = 0; i < N; ++i) on[i] = nb[i] >= 0 && ((now >> k[i]) & 1u);
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (on[i]) de.add(nb[i], x[i]);
        __syncwarp();
        rest &= ~now;
    }
    if (!rest) return;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool on = nb[i] >= 0 && ((rest >> k[i]) & 1u);
        const unsigned grp = __match_any_sync(kFull, on ? nb[i] : -1 - (int)lane);
        const bool alone = grp == (1u << lane);
        if (on && alone) de.add(nb[i], x[i]);
        if (__any_sync(kFull, on && !alone)) {
            scratch[lane] = x[i];
            __syncwarp();
            if (on && !alone && lane == (unsigned)(__ffs(grp) - 1))
                add_group(de, nb[i], grp, scratch);
        }
        __syncwarp();
    }
}

// The neighbour updates of every lane whose bit is set in `fm`: slot x gets
// (mult * J) * val(x) for each entry (x, J) of the lane's list.  Lane k of the
// warp holds its variable v, list start `start`, degree `deg` and factor
// `mult` (valid on flipping lanes).  The flipping variables must be pairwise
// non-adjacent.  Entries are applied lane-parallel in rounds of 32; equal
// targets within a round are summed in entry order by their first lane.
// `scratch` holds 32 doubles followed by 32 ints.
// WINDOWED: the lanes are the variables of one window, and entries naming a
// later variable of it are left out.
// REG: lists of one length.
// PHASED: in global slots, lists of different lengths whose flips may share
// neighbours go in phases (add_phased) instead of being matched 32 entries at
// a time: 500 reads x 20 Gibbs sweeps of a sparse n = 4000, degree 12 problem
// 7.0 -> 6.2 ms.  (Slower so: equal lists, 2% on the uneven batch, and state in
// shared memory, n = 400, 5%.)
template <bool REG, bool WINDOWED = false, bool PHASED = false, class DE, class VAL>
__device__ __forceinline__ void push_entries(const Prob &P, DE de, VAL val,
                                             double *scratch, unsigned fm, int v,
                                             int start, int deg, double mult,
                                             bool may_conflict, unsigned lane, uint32_t shr = 0u) {
    const bool f = (fm >> lane) & 1u;
    [[maybe_unused]] const int w0 = v - (int)lane;
    int *owner_of_rank = reinterpret_cast<int *>(scratch + 32);
    const int D = REG ? P.regular_degree : 0;
    int excl = 0, total;
    if constexpr (REG) {
        // Equal list lengths: entry t belongs to the (t / D)-th flip.
        if (f) owner_of_rank[__popc(fm & ((1u << lane) - 1u))] = (int)lane;
        total = __popc(fm) * D;
        __syncwarp();
    } else {
        const int my = f ? deg : 0;
        int incl = my;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if ((int)lane >= o) incl += y;
        }
        excl = incl - my;
        total = __shfl_sync(kFull, incl, 31);
    }
    // (shr bit 0: a list names a target twice.)
    const bool phased = PHASED && DE::kAsyncAdd && may_conflict && !REG &&
                        !__any_sync(kFull, f && (shr & 1u));
    if (!REG && (!may_conflict || phased)) {
        // No two entries name the same slot: each chunk of 96 entries issues
        // all of its delta-energy loads before its stores.
        for (int base = 0; base < total; base += 96) {
            int nb[3], kk[3];
            double x[3], dv[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int t = base + 32 * i + (int)lane;
                int k = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    const int ex = __shfl_sync(kFull, excl, k + step);
                    if (ex <= t) k += step;
                }
                const int e = __shfl_sync(kFull, start, k) + (t - __shfl_sync(kFull, excl, k));
                const double m_k = __shfl_sync(kFull, mult, k);
                kk[i] = k;
                nb[i] = -1;
                x[i] = 0.0;
                if (t < total) {
                    nb[i] = __ldg(&P.col[e]);
                    x[i] = __dmul_rn(__dmul_rn(m_k, __ldg(&P.w[e])), val(nb[i]));
                    if (WINDOWED && nb[i] > w0 + k && nb[i] < w0 + 32) nb[i] = -1;
                }
            }
            if (PHASED && DE::kAsyncAdd && phased) {
                add_phased<3>(de, nb, x, kk, fm, shr, scratch, lane);
            } else if constexpr (DE::kAsyncAdd) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (nb[i] >= 0) de.add(nb[i], x[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (nb[i] >= 0) dv[i] = de.get(nb[i]);
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (nb[i] >= 0) de.set(nb[i], __dadd_rn(dv[i], x[i]));
            }
        }
        __syncwarp();
        total = 0;  // done
    }
    for (int base = 0; base < total; base += 32) {
        const int t = base + (int)lane;
        bool a = t < total;
        int k, e;
        if constexpr (REG) {
            const int r = (int)(((uint32_t)t * P.regular_magic) >> 16);  // t / D
            k = a ? owner_of_rank[r] : 0;
            e = __shfl_sync(kFull, v, k) * D + (t - r * D);
        } else {
            // Owner: the last lane whose entry range starts at or before t.
            k = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int ex = __shfl_sync(kFull, excl, k + step);
                if (ex <= t) k += step;
            }
            e = __shfl_sync(kFull, start, k) + (t - __shfl_sync(kFull, excl, k));
        }
        const double m_k = __shfl_sync(kFull, mult, k);
        int nb = -1 - (int)lane;  // distinct per inactive lane
        double x = 0.0;
        if (a) {
            nb = __ldg(&P.col[e]);
            x = __dmul_rn(__dmul_rn(m_k, __ldg(&P.w[e])), val(nb));
            if (WINDOWED && nb > w0 + k && nb < w0 + 32) a = false, nb = -1 - (int)lane;
        }
        const unsigned grp = may_conflict ? __match_any_sync(kFull, nb) : (1u << lane);
        const bool alone = grp == (1u << lane);
        if (a && alone) de.add(nb, x);
        if (may_conflict && __any_sync(kFull, a && !alone)) {
            scratch[lane] = x;
            __syncwarp();
            if (a && !alone && lane == (unsigned)(__ffs(grp) - 1)) {
                add_group(de, nb, grp, scratch);
            }
        }
        __syncwarp();
    }
}

// cpu_sa.cpp:168-191 for the flips `fm` (see push_entries); `s_old` is the
// lane's spin.  With `own_fresh`, no entry of this pass names the lane's own
// slot, which then still holds `d_own`.
template <bool REG, bool PHASED = false, class DE>
__device__ __forceinline__ void apply_flips(const Prob &P, DE de, int8_t *sp,
                                            double *scratch, unsigned fm, int v,
                                            int start, int deg, int s_old,
                                            bool may_conflict, unsigned lane,
                                            bool own_fresh = false, double d_own = 0.0,
                                            uint32_t shr = 0u) {
    push_entries<REG, false, PHASED>(P, de, [&](int x) { return (double)(int)sp[x]; }, scratch, fm, v, start, deg,
                 (double)(int)(int8_t)(4 * s_old), may_conflict, lane, shr);
    if ((fm >> lane) & 1u) {  // cpu_sa.cpp:189-190, after the variable's own updates
        sp[v] = (int8_t)(-s_old);
        de.set(v, __dmul_rn(own_fresh ? d_own : de.get(v), -1.0));
    }
    __syncwarp();
}

// Adjacency entries t = 32 i + lane (i < kPreGroups) of the accepted flips'
// lists in flip order, loaded before the commit point is known: target,
// coupling and the lane of the entry's flip.
constexpr int kPreGroups = 2;
struct PreEntries {
    int nb[kPreGroups];
    int k[kPreGroups];
    double w[kPreGroups];
};

// Entry t of the flips' lists for equal-length lists (list v at v * D): its
// target, coupling and the lane k of its flip.  `rank_tab[f]` is the lane of
// the f-th flip in variable order.  STAGED: P.col and P.w hold the lists of
// this window alone, in shared memory.
template <bool STAGED = false>
__device__ __forceinline__ void regular_load(const Prob &P, const int *rank_tab, int p, int t,
                                             int &k, int &nb, double &wt) {
    const int D = P.regular_degree;
    const int r = (int)(((uint32_t)t * P.regular_magic) >> 16);  // t / D
    k = rank_tab[r];
    if constexpr (STAGED) {
        const int e = k * D + (t - r * D);
        nb = P.col[e];
        wt = P.w[e];
    } else {
        const int e = (p + k) * D + (t - r * D);
        nb = __ldg(&P.col[e]);
        wt = __ldg(&P.w[e]);
    }
}

// Neighbour updates of the committed flips for equal-length lists.  `mult` is
// each lane's (int8)(4 * s) as a double (cpu_sa.cpp:172), read from the
// entry's owner lane.  With `pre`, the first 32 kPreGroups entries are in `pe`
// (loaded when only the accepted flips were known; the committed flips are a
// prefix of them); the other entries are loaded here.
//
// When no two entries of the pass can name the same slot, the entries go in
// chunks of 32 kPreGroups whose delta-energy loads are all issued before
// their stores, so a chunk waits on memory once.  Otherwise they go in rounds
// of 32, equal targets within a round summed in entry order by their first
// lane, as in apply_flips.  WINDOWED: entries naming a later variable of the
// window are left out.
template <bool WINDOWED = false, bool STAGED = false, class DE>
__device__ __forceinline__ void update_regular(const Prob &P, DE de, const int8_t *sp,
                                               double *scratch, const int *rank_tab,
                                               int nflips, int p, bool pre, const PreEntries &pe,
                                               bool may_conflict, double mult, unsigned lane) {
    const int total = nflips * P.regular_degree;
    if (!may_conflict) {
        for (int base = 0; base < total; base += 32 * kPreGroups) {
            int nb[kPreGroups];
            double x[kPreGroups], dv[kPreGroups];
#pragma unroll
            for (int i = 0; i < kPreGroups; ++i) {
                const int t = base + 32 * i + (int)lane;
                int k = 0, q = 0;
                double wt = 0.0;
                if (pre && base == 0) {
                    k = pe.k[i], q = pe.nb[i], wt = pe.w[i];
                } else if (t < total) {
                    regular_load<STAGED>(P, rank_tab, p, t, k, q, wt);
                }
                const double m_k = __shfl_sync(kFull, mult, k);
                x[i] = __dmul_rn(__dmul_rn(m_k, wt), (double)(int)sp[q]);
                nb[i] = t >= total || (WINDOWED && q > p + k && q < p + 32) ? -1 : q;
            }
            if constexpr (DE::kAsyncAdd) {
#pragma unroll
                for (int i = 0; i < kPreGroups; ++i)
                    if (nb[i] >= 0) de.add(nb[i], x[i]);
            } else {
#pragma unroll
                for (int i = 0; i < kPreGroups; ++i)
                    if (nb[i] >= 0) dv[i] = de.get(nb[i]);
#pragma unroll
                for (int i = 0; i < kPreGroups; ++i)
                    if (nb[i] >= 0) de.set(nb[i], __dadd_rn(dv[i], x[i]));
            }
        }
        __syncwarp();
        return;
    }
    for (int base = 0; base < total; base += 32) {
        const int t = base + (int)lane;
        bool a = t < total;
        int k = 0, nb = 0;
        double wt = 0.0;
        if (pre && base == 0) {
            k = pe.k[0], nb = pe.nb[0], wt = pe.w[0];
        } else if (pre && base == 32) {
            k = pe.k[1], nb = pe.nb[1], wt = pe.w[1];
        } else if (a) {
            regular_load<STAGED>(P, rank_tab, p, t, k, nb, wt);
        }
        const double m_k = __shfl_sync(kFull, mult, k);
        double x = 0.0;
        if (a) {
            x = __dmul_rn(__dmul_rn(m_k, wt), (double)(int)sp[nb]);
            if (WINDOWED && nb > p + k && nb < p + 32) a = false;
        }
        if (!a) nb = -1 - (int)lane;  // distinct per inactive lane
        const unsigned grp = __match_any_sync(kFull, nb);
        const bool alone = grp == (1u << lane);
        if (a && alone) de.add(nb, x);
        if (__any_sync(kFull, a && !alone)) {
            scratch[lane] = x;
            __syncwarp();
            if (a && !alone && lane == (unsigned)(__ffs(grp) - 1)) {
                add_group(de, nb, grp, scratch);
            }
        }
        __syncwarp();
    }
}

// One acceptance decision (cpu_sa.cpp:144-166) for a lane that needs a draw:
// the single-precision bounds first, the exact double test inside the band.
// Returns accept in bit 0 and the near-tie flag in bit 1.
template <bool GIBBS>
__device__ __forceinline__ int decide(double d, double beta, uint64_t r) {
    const int fast = GIBBS ? gibbs_fast(__dmul_rn(d, beta), r)
                           : metropolis_fast(__dmul_rn(-d, beta), r);
    if (fast >= 0) return fast;
    return GIBBS ? gibbs_exact(d, beta, r) : metropolis_exact(d, beta, r);
}

// log2 of a draw for the acceptance bounds, from its upper half: truncation
// and rounding stay below 2^-18 for draws of 2^52 and more; smaller ones
// (2^-12 of all) give NaN, which leaves the decision to the exact test.
__device__ __forceinline__ float draw_log2(uint64_t r) {
    const uint32_t hi = (uint32_t)(r >> 32);
    const float y = lg2_approx(__uint2float_rn(hi)) + 32.0f;
    return hi >= (1u << 20) ? y : __int_as_float(0x7fffffff);
}

// A lane's decision on its delta energy d (cpu_sa.cpp:140-166): whether it
// draws, and the bound t that the log2 of an accepted draw stays below (see
// metropolis_fast and gibbs_fast): +inf for a flip without a draw, -inf for
// none.  The bound is taken from d in single precision, which adds two roundings
// of a product below 64; betas beyond the range of that give NaN, which leaves
// every decision to the exact test.
template <bool GIBBS>
struct Choice {
    bool need;
    float t;

    // Per beta: beta log2(e), the factor of d.
    static __device__ __forceinline__ float scale(double beta) {
        return beta == 0.0 || (beta > 1e-30 && beta < 1e30) ? (float)(beta * (double)kLog2e)
                                                            : __int_as_float(0x7fffffff);
    }
    __device__ __forceinline__ void look(double d, float scale, double thr, bool act) {
        const float inf = __int_as_float(0x7f800000);
        const bool cons = act && !(d >= thr);
        const float z = (float)d * scale;  // log2(exp(d * beta))
        if constexpr (GIBBS) {
            need = cons;
            // log2(1 + exp(z)), see gibbs_fast
            const float big = 24.0f * kLog2e;
            const float g = z > big ? z : z < -big ? 0.0f : lg2_approx(1.0f + ex2_approx(z));
            t = cons ? 64.0f - g : -inf;
        } else {
            const bool down = d <= 0.0;
            need = cons && !down;
            t = !cons ? -inf : down ? inf : 64.0f - z;
        }
    }
    // The exact decision.  Bit 0: flips, bit 1: near tie.
    __device__ __forceinline__ int exact(double d, double beta, uint64_t r) const {
        if (!need) return t > 0.0f ? 1 : 0;
        return GIBBS ? gibbs_exact(d, beta, r) : metropolis_exact(d, beta, r);
    }
};

// Sequential order (cpu_sa.cpp:132-192) in speculative passes over windows
// of 32 consecutive variables, one per lane.  Every lane decides its variable
// against the delta energies at the start of the pass; the pass commits the
// prefix of the window that ends before the first variable whose decision a
// committed flip could have changed (a later neighbour of an accepted flip),
// so the committed decisions equal the sequential ones.
//
// While a window is processed, the records of the next one are prefetched
// into L1 when the delta energies are on chip or in the band.
//
// BANDED (kStageBand): the delta energies of variables within band_b of the
// window live in a shared-memory ring of band_w slots (BandDe), the rest in
// the global slot `de_g`.  After each pass the band slides by the committed
// count: the slots leaving it are written back and the ones entering are
// fetched asynchronously.  band_w >= 2 band_b + 128 keeps the slots fetched
// by a slide at least four passes ahead of the window, so every pass waits
// only for the slides before the last one (cp.async.wait_group 1) before its
// decisions read the window; an update through a coupler longer than band_b
// can reach the last slide's slots, so the update phase waits for all of
// them.  At every sweep the band is written back and reloaded from the start.
//
// The band at the start of a sweep: written back (when `live`) and reloaded
// around variable 0.
__device__ __forceinline__ void band_rewind(BandDe &de, int n, int band_b, bool live,
                                            unsigned lane) {
    cp_async_wait<0>();
    __syncwarp();
    const int w = (int)de.w;
    const unsigned mask = de.w - 1u;
    if (live) {
        for (int i = (int)lane; i < w; i += 32) {
            const int x = de.lo + i;
            if (x >= 0 && x < n) de.g[x] = de.b[(unsigned)x & mask];
        }
        __syncwarp();
    }
    de.lo = -band_b;
    const int top = min(n, w - band_b);
    for (int x = (int)lane; x < top; x += 32) de.b[(unsigned)x & mask] = de.g[x];
    __syncwarp();
}

// The band after a pass over the window at p that committed c variables.
__device__ __forceinline__ void band_slide(const BandDe &de, int n, int p, int band_b, int c,
                                           unsigned lane) {
    __syncwarp();
    if ((int)lane < c) {
        const int xo = p - band_b + (int)lane;  // < p: band_b >= 32
        const unsigned slot = (unsigned)xo & (de.w - 1u);
        if (xo >= 0) de.g[xo] = de.b[slot];
        const int xn = xo + (int)de.w;
        if (xn < n) cp_async8(&de.b[slot], &de.g[xn]);
    }
    cp_async_commit();
    __syncwarp();
}

template <bool GIBBS, int STAGE, bool REG>
__device__ __forceinline__ void sweep_sequential(const Prob &P, double *de_g,
                                                 int8_t *sp, double *scratch,
                                                 uint64_t *ring, RingState &rs,
                                                 unsigned lane, double *band, int band_w,
                                                 int band_b) {
    constexpr bool BANDED = STAGE == kStageBand;
    const int n = P.n;
    const int D = REG ? P.regular_degree : 0;
    const unsigned lt_mask = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7f800000);
    int *rank_tab = reinterpret_cast<int *>(scratch + 32);
    typename DeFor<STAGE>::T de;
    bool band_live = false;
    if constexpr (BANDED)
        de = BandDe{de_g, band, 0, (unsigned)band_w};
    else
        de.p = de_g;
    for (int b = 0; b < reload(P.pd->num_betas); ++b) {
        const double beta = __ldg(&reload(P.pd->betas)[b]);
        const double thr = __ldg(&reload(P.pd->thresholds)[b]);
        const float scale = Choice<GIBBS>::scale(beta);
        for (int sw = 0; sw < reload(P.pd->sweeps_per_beta); ++sw) {
            SweepCount cnt;
            if constexpr (BANDED) {
                if (band_w) band_rewind(de, n, band_b, band_live, lane);
                band_live = true;
            }
            int p = 0;
            while (p < n) {
                if constexpr (BANDED) {
                    if (band_w) {  // the slides of all but the last pass have landed
                        cp_async_wait<1>();
                        __syncwarp();
                    }
                }
                ring_refill(ring, rs, lane);
                const int L = min(32, n - p);
                const int v = p + (int)lane;
                const bool act = (int)lane < L;
                double d = 0.0;
                int dist = (int)kDistCap;
                uint32_t shr = 0u;
                uint2 vi = make_uint2(0u, 0u);
                int s_cur = 0;
                if (act) {
                    d = de.get(v);
                    dist = __ldg(&P.dist[v]);
                    shr = __ldg(&P.share[v]);
                    if (!REG) vi = __ldg(&P.vinfo[v]);
                    s_cur = (int)sp[v];
                }
                if (act) {
                    // The next window starts at p + c <= p + 32 and ends
                    // before p + c + 32, so the lines of [v + 32] are the
                    // ones it may need beyond this window's.
                    const int vn = v + 32;
                    // (Not with global slots: there the prefetches measured
                    // slower than the plain loads.)
                    if (vn < n && !DeFor<STAGE>::T::kAsyncAdd) {
                        prefetch_l1(P.dist + vn);
                        prefetch_l1(P.share + vn);
                        if (!REG) prefetch_l1(P.vinfo + vn);
                    }
                }
                // cpu_sa.cpp:140-166.  (All lanes take a draw's logarithm and
                // compare; a branch for those that need one measured 2-3%
                // slower on the uneven batch.)
                Choice<GIBBS> ch;
                ch.look(d, scale, thr, act);
                const unsigned nm = __ballot_sync(kFull, ch.need);
                unsigned am = 0u, ties = 0u;
                // (A bound of NaN counts as a decision to be made.)
                if (__any_sync(kFull, !(ch.t == -inf))) {
                    const int at = __popc(nm & lt_mask);
                    const float y = draw_log2(ring[(rs.q + lane) & (kRing - 1)]);
                    const float gap = ch.t - __shfl_sync(kFull, y, at);
                    am = __ballot_sync(kFull, gap > kBand);
                    if (__any_sync(kFull, !(fabsf(gap) > kBand))) {  // inside the band
                        int x = 0;
                        if (!(fabsf(gap) > kBand))
                            x = ch.exact(d, beta, ring[(rs.q + (uint32_t)at) & (kRing - 1)]);
                        am |= __ballot_sync(kFull, (x & 1) != 0);
                        ties = __ballot_sync(kFull, (x & 2) != 0);
                    }
                }
                const bool acc = (am >> lane) & 1u;
                // Equal-length lists: start loading the accepted flips'
                // adjacency before the commit point is known.
                const double mult = (double)(int)(int8_t)(4 * s_cur);
                PreEntries pe;
#pragma unroll
                for (int i = 0; i < kPreGroups; ++i) pe.nb[i] = 0, pe.k[i] = 0, pe.w[i] = 0.0;
                if (REG && am) {
                    if (acc) rank_tab[__popc(am & lt_mask)] = (int)lane;
                    __syncwarp();
                    const int pre_n = min(__popc(am) * D, 32 * kPreGroups);
#pragma unroll
                    for (int i = 0; i < kPreGroups; ++i) {
                        const int t = (int)lane + 32 * i;
                        if (t < pre_n) regular_load(P, rank_tab, p, t, pe.k[i], pe.nb[i], pe.w[i]);
                    }
                }
                const int bound = acc ? (int)lane + dist : 32;
                const int c = am ? min(__reduce_min_sync(kFull, bound), L) : L;
                const unsigned done = c >= 32 ? kFull : ((1u << c) - 1u);
                const unsigned fm = am & done;
                rs.q += (uint32_t)__popc(nm & done);
                cnt.pass((unsigned)__popc(fm), (unsigned)__popc(ties & done));
                if constexpr (BANDED) {
                    // The slots the last slide fetched lie at the far end of
                    // the band, which only an update through a coupler longer
                    // than band_b can reach: they land before the update phase.
                    if (band_w && fm) {
                        cp_async_wait<0>();
                        __syncwarp();
                    }
                }
                if (fm) {
                    // A slot can receive two additions only through a repeated
                    // target in one list or a neighbour common to two flips.
                    const unsigned later = lane < 31 ? fm >> (lane + 1) : 0u;
                    const bool f = (fm >> lane) & 1u;
                    const bool may_conflict =
                        __any_sync(kFull, f && ((shr & 1u) || ((shr >> 1) & later)));
                    // The committed flips are pairwise non-adjacent, so a
                    // flip's own slot receives an addition in this pass only
                    // from a repeated target in its own list; otherwise it
                    // still holds the window value d and the negation needs no
                    // load.
                    const bool own_fresh = !(shr & 1u);
                    if constexpr (REG) {
                        update_regular(P, de, sp, scratch, rank_tab, __popc(fm), p, true, pe,
                                       may_conflict, mult, lane);
                        if (f) {  // cpu_sa.cpp:189-190, after the variable's own updates
                            sp[v] = (int8_t)(-s_cur);
                            de.set(v, __dmul_rn(own_fresh ? d : de.get(v), -1.0));
                        }
                        __syncwarp();
                    } else {
                        apply_flips<REG, true>(P, de, sp, scratch, fm, v, (int)vi.x,
                                               (int)(vi.y & kDegMask), s_cur, may_conflict, lane,
                                          own_fresh, d, shr);
                    }
                }
                if constexpr (BANDED) {
                    if (band_w) band_slide(de, n, p, band_b, c, lane);
                }
                p += c;
                if constexpr (BANDED) de.lo = p - band_b;
            }
            cnt.flush(ring, lane);
        }
    }
    if constexpr (BANDED) {
        if (band_w) {  // nothing of this read may land after it
            cp_async_wait<0>();
            __syncwarp();
        }
    }
}

// Sequential order for problems whose window variables often neighbour each
// other (`resolve`: lists name no target twice), on reads whose spins are all
// +-1.  Every pass commits its whole window.
//
// The decisions of a window solve a recursion: lane k's delta energy is the one
// at the start of the pass plus ((4 s_j) J) s_k of every flipped lane j < k it
// neighbours, in variable order (cpu_sa.cpp:172-185), and its draw is placed
// after those of the drawing lanes before it.  The lanes solve it together:
// from an assumed set of flips all of them decide at once, the flips that come
// out are the next assumption, until a set reproduces itself.  A lane's
// decision depends on earlier lanes only, so after i rounds at least the first
// i lanes are as in the reference, and the set that reproduces itself is the
// reference's.  Changes die out quickly, so rounds are few.  (Committing up to
// the first dependent lane per round and deciding the rest anew took about one
// round per dependent flip: L = 32 lattice, 256 reads x 64 sweeps 226 -> 171 ms;
// L = 8, 4096 x 50 5.0 -> 3.4; L = 16, 1000 x 20 11.9 -> 7.4.)
//
// The update phase writes the window's own delta energies and spins first: they
// hold the contributions of the earlier flips and the variable's own negation.
// Then it applies every flip's other entries in variable order: those naming
// an earlier variable of the window or one outside it.
//
// Delta energies on chip or in the band: the next window's records are loaded
// into registers while this one is worked on (a window always starts 32
// further on).
template <bool GIBBS, int STAGE, bool REG>
__device__ __forceinline__ void sweep_resolved(const Prob &P, double *de_g, int8_t *sp,
                                               double *scratch, uint64_t *ring, RingState &rs,
                                               unsigned lane, double *band, int band_w,
                                               int band_b) {
    constexpr bool BANDED = STAGE == kStageBand;
    constexpr bool AHEAD = !DeFor<STAGE>::T::kAsyncAdd;
    const int n = P.n;
    const int D = REG ? P.regular_degree : 0;
    const unsigned lt_mask = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7f800000);
    int *rank_tab = reinterpret_cast<int *>(scratch + 32);
    typename DeFor<STAGE>::T de;
    bool band_live = false;
    if constexpr (BANDED)
        de = BandDe{de_g, band, 0, (unsigned)band_w};
    else
        de.p = de_g;
    // A variable's records.  `near` is the coupling of the nearest back
    // neighbour (stored last), on lattices and chains the one that matters.
    struct Record {
        uint32_t shr;
        uint2 vi, bk;
        double near;
    };
    auto load = [&](int v) {
        Record r{0u, make_uint2(0u, 0u), make_uint2(0u, 0u), 0.0};
        if (v < n) {
            r.shr = __ldg(&P.wshare[v]);
            r.vi = REG ? make_uint2((uint32_t)v * (uint32_t)D, (uint32_t)D) : __ldg(&P.vinfo[v]);
            r.bk = __ldg(&P.back[v]);
        }
        return r;
    };
    auto load_near = [&](Record &r) {
        if (r.bk.x) r.near = __ldg(&P.bw[r.bk.y + (uint32_t)__popc(r.bk.x) - 1u]);
    };
    Record next = load((int)lane);
    load_near(next);
    // Equal lists and a band: the next window's lists (whole 16-byte pieces)
    // are copied into one of two buffers behind the band while this window is
    // worked on; they land with the band's next slide.  (Loads of them in the
    // update phase waited on L2, a quarter of the pass: prefetch.global.L1 does
    // not bring a line into L1 here.  With the left-out entries, which remove
    // most conflicts, L = 32, 256 reads x 64 sweeps 171 -> 147 ms, L = 16, 1000 x
    // 20 7.4 -> 6.4.)
    [[maybe_unused]] const bool staged = BANDED && REG && band_w > 0 && D <= kListMaxDegree;
    [[maybe_unused]] double *list_w = band + band_w;
    [[maybe_unused]] int32_t *list_col =
        reinterpret_cast<int32_t *>(list_w + 2 * 32 * kListMaxDegree);
    [[maybe_unused]] auto stage = [&](int p) {
        const int entries = min(32, n - p) * D;
        const double *w = P.w + (int64_t)p * D;
        const int32_t *col = P.col + (int64_t)p * D;
        double *to_w = list_w + (p & 32) * D;
        int32_t *to_col = list_col + (p & 32) * D;
        for (int i = (int)lane; 2 * i < entries; i += 32) cp_async16(to_w + 2 * i, w + 2 * i);
        for (int i = (int)lane; 4 * i < entries; i += 32) cp_async16(to_col + 4 * i, col + 4 * i);
    };
    if constexpr (BANDED) {
        if (staged) {
            stage(0);
            cp_async_commit();
        }
    }
    for (int b = 0; b < reload(P.pd->num_betas); ++b) {
        const double beta = __ldg(&reload(P.pd->betas)[b]);
        const double thr = __ldg(&reload(P.pd->thresholds)[b]);
        const float scale = Choice<GIBBS>::scale(beta);
        for (int sw = 0; sw < reload(P.pd->sweeps_per_beta); ++sw) {
            SweepCount cnt;
            if constexpr (BANDED) {
                if (band_w) band_rewind(de, n, band_b, band_live, lane);
                band_live = true;
            }
            for (int p = 0; p < n; p += 32) {
                if constexpr (BANDED) {
                    if (band_w) {  // the slides of all but the last pass have landed
                        cp_async_wait<1>();
                        __syncwarp();
                    }
                }
                ring_refill(ring, rs, lane);
                const int v = p + (int)lane;
                const bool act = v < n;
                double d0 = 0.0;
                int s_cur = 0;
                if (act) {
                    d0 = de.get(v);
                    s_cur = (int)sp[v];
                }
                Record r;
                if constexpr (AHEAD) {
                    r = next;
                    const int vn = p + 32 < n ? v + 32 : (int)lane;
                    next = load(vn);
                    if constexpr (BANDED) {
                        if (staged && p + 32 < n) stage(p + 32);
                    }
                } else {
                    r = load(v);
                    load_near(r);
                }
                double d = d0;
                unsigned rel = 0u;  // flipped lanes before this one, as d holds them
                Choice<GIBBS> ch;
                ch.look(d, scale, thr, act);
                unsigned fm = 0u, ties = 0u;
                // (A bound of NaN counts as a decision to be made.)
                if (__any_sync(kFull, !(ch.t == -inf))) {
                    const float y = draw_log2(ring[(rs.q + lane) & (kRing - 1)]);
                    // Lanes before this one whose variables neighbour its own.
                    const unsigned back = act ? __brev(r.bk.x) >> (31u - lane) : 0u;
                    const int o_near = r.bk.x ? __ffs(r.bk.x) - 1 : 0;
                    const unsigned up = __ballot_sync(kFull, s_cur > 0);
                    unsigned nm;
                    for (;;) {
                        nm = __ballot_sync(kFull, ch.need);
                        const int at = __popc(nm & lt_mask);
                        const float gap = ch.t - __shfl_sync(kFull, y, at);
                        fm = __ballot_sync(kFull, gap > kBand);
                        ties = 0u;
                        if (__any_sync(kFull, !(fabsf(gap) > kBand))) {  // inside the band
                            int x = 0;
                            if (!(fabsf(gap) > kBand))
                                x = ch.exact(d, beta, ring[(rs.q + (uint32_t)at) & (kRing - 1)]);
                            fm |= __ballot_sync(kFull, (x & 1) != 0);
                            ties = __ballot_sync(kFull, (x & 2) != 0);
                        }
                        const bool changed = (back & fm) != rel;
                        if (!__any_sync(kFull, changed)) break;
                        if (changed) {
                            rel = back & fm;
                            d = d0;
                            for (unsigned m = rel; m; m &= m - 1u) {
                                const int j = __ffs(m) - 1;
                                const int o = (int)lane - j;
                                double wj = r.near;
                                if (o != o_near)  // offsets are stored descending
                                    wj = __ldg(&P.bw[r.bk.y +
                                                     (uint32_t)__popc((r.bk.x >> o) >> 1)]);
                                // ((4 s_j) J) s_k, exactly +-4 J
                                const bool same = (((up >> j) & 1u) != 0u) == (s_cur > 0);
                                d = __dadd_rn(d, __dmul_rn(wj, same ? 4.0 : -4.0));
                            }
                            ch.look(d, scale, thr, act);
                        }
                    }
                    rs.q += (uint32_t)__popc(nm);
                }
                cnt.pass((unsigned)__popc(fm), (unsigned)__popc(ties));
                if (fm) {
                    if constexpr (BANDED) {
                        // The slots the last slide fetched lie at the far end
                        // of the band, which only an update through a coupler
                        // longer than band_b can reach: they land before the
                        // update phase.
                        if (band_w) {
                            cp_async_wait<0>();
                            __syncwarp();
                        }
                    }
                    // A slot can receive two of the additions below only
                    // through a neighbour common to two flips.
                    const unsigned later = lane < 31 ? fm >> (lane + 1) : 0u;
                    const bool f = (fm >> lane) & 1u;
                    const bool may_conflict = __any_sync(kFull, f && ((r.shr >> 1) & later));
                    // cpu_sa.cpp:189-190, the contributions of the window's
                    // earlier flips included.
                    if (f || rel) de.set(v, f ? -d : d);
                    if (f) sp[v] = (int8_t)(-s_cur);
                    const double mult = (double)(4 * s_cur);
                    if constexpr (REG) {
                        if (f) rank_tab[__popc(fm & lt_mask)] = (int)lane;
                        __syncwarp();
                        const PreEntries none{};
                        if (BANDED && staged) {
                            Prob W = P;
                            W.col = list_col + (p & 32) * D;
                            W.w = list_w + (p & 32) * D;
                            update_regular<true, BANDED>(W, de, sp, scratch, rank_tab, __popc(fm),
                                                         p, false, none, may_conflict, mult, lane);
                        } else {
                            update_regular<true>(P, de, sp, scratch, rank_tab, __popc(fm), p,
                                                 false, none, may_conflict, mult, lane);
                        }
                    } else {
                        __syncwarp();
                        push_entries<REG, true, true>(P, de, [&](int x) { return (double)(int)sp[x]; },
                                           scratch, fm, v, (int)r.vi.x, (int)(r.vi.y & kDegMask),
                                           mult, may_conflict, lane, r.shr);
                    }
                }
                if constexpr (BANDED) {
                    // (Window 0's buffer may be this last window's.)
                    if (staged && p + 32 >= n) {
                        __syncwarp();
                        stage(0);
                    }
                    const int c = min(32, n - p);
                    if (band_w) band_slide(de, n, p, band_b, c, lane);
                    de.lo = p + c - band_b;
                }
                if constexpr (AHEAD) load_near(next);
            }
            cnt.flush(ring, lane);
        }
    }
    if constexpr (BANDED) {
        if (band_w) {  // nothing of this read may land after it
            cp_async_wait<0>();
            __syncwarp();
        }
    }
}

// rv % n (cpu_sa.cpp:135) with magic = (2^64 - 1) / n: the estimated quotient
// is at most one too small.
__device__ __forceinline__ int mod_n(uint64_t rv, uint32_t n, uint64_t magic) {
    const uint64_t r = rv - __umul64hi(rv, magic) * (uint64_t)n;
    return (int)(uint32_t)(r >= n ? r - n : r);
}

// Lists up to this long are scanned by their own lane for the window's
// accepted variables (random_commit; regular degree 6, n = 500, 50 sweeps in random order: 6.3 -> 4.3 ms; lists of
// 15 on average 14.3 -> 13.7, of 40 unchanged at 15.0).
constexpr int kScanDegree = 16;

// The commit point of a window in random order: the first chain lane whose
// variable an earlier accepted lane (bit of A) flipped or neighbours; 32 when
// there is none.  `touch` is a bitmap of the variables, clear before and after.
//
// Short lists: the accepted lanes mark their variables all at once and every
// chain lane looks for a mark in its own list, so a window without a hit (the
// usual one on a sparse graph) costs one scan, whatever the number of
// accepted lanes.
// Long lists: the accepted lanes mark their neighbours one after another, the
// list spread over the warp.
__device__ __forceinline__ int random_commit(const Prob &P, int D, uint32_t *touch, int var,
                                             bool chain, unsigned A, unsigned lane) {
    if (!A) return 32;
    const uint2 own = D ? make_uint2((uint32_t)var * (uint32_t)D, (uint32_t)D)
                        : __ldg(&P.vinfo[var]);
    const unsigned deg_own = own.y & kDegMask;
    const bool acc = (A >> lane) & 1u;
    int c = 32;
    if (__all_sync(kFull, !chain || deg_own <= (unsigned)kScanDegree)) {
        if (acc) atomicOr(&touch[var >> 5], 1u << (var & 31));
        __syncwarp();
        bool near = false;
        for (unsigned t = 0; chain && t < deg_own; ++t) {
            const int x = __ldg(&P.col[own.x + t]);
            near = near || ((touch[x >> 5] >> (x & 31)) & 1u);
        }
        const unsigned lt_mask = (1u << lane) - 1u;
        const bool again = (__match_any_sync(kFull, var) & A & lt_mask) != 0u;
        __syncwarp();
        if (acc) touch[var >> 5] = 0u;
        const unsigned H = __ballot_sync(kFull, chain && again);
        if (H) c = __ffs(H) - 1;
        // Lanes next to an accepted one, lowest first: the first of them with
        // an earlier such neighbour is the commit point.
        for (unsigned M = __ballot_sync(kFull, chain && near); M; M &= M - 1u) {
            const int l = __ffs(M) - 1;
            if (l >= c) break;
            const unsigned start = __shfl_sync(kFull, own.x, l), deg = __shfl_sync(kFull, deg_own, l);
            bool hit = false;
            for (unsigned t = 0; t < deg; ++t) hit = hit || __ldg(&P.col[start + t]) == var;
            if (__ballot_sync(kFull, hit) & A & ((1u << l) - 1u)) c = l;
        }
        __syncwarp();
        return c;
    }
    unsigned todo = A, marked = 0u;
    while (todo) {
        const int j = __ffs(todo) - 1;
        if (j >= c) break;
        todo &= todo - 1u;
        marked |= 1u << j;
        const int vj = __shfl_sync(kFull, var, j);
        const unsigned start = __shfl_sync(kFull, own.x, j), deg = __shfl_sync(kFull, deg_own, j);
        for (unsigned t = lane; t < deg; t += 32) {
            const int x = __ldg(&P.col[start + t]);
            atomicOr(&touch[x >> 5], 1u << (x & 31));
        }
        if (lane == 0) atomicOr(&touch[vj >> 5], 1u << (vj & 31));
        __syncwarp();
        const bool hit = chain && (int)lane > j && ((touch[var >> 5] >> (var & 31)) & 1u);
        const unsigned H = __ballot_sync(kFull, hit);
        if (H) c = min(c, __ffs(H) - 1);
    }
    __syncwarp();
    for (unsigned m = marked; m; m &= m - 1u) {  // clear the marked words for the next pass
        const int j = __ffs(m) - 1;
        const int vj = __shfl_sync(kFull, var, j);
        const unsigned start = __shfl_sync(kFull, own.x, j), deg = __shfl_sync(kFull, deg_own, j);
        for (unsigned t = lane; t < deg; t += 32) touch[__ldg(&P.col[start + t]) >> 5] = 0u;
        if (lane == 0) touch[vj >> 5] = 0u;
    }
    __syncwarp();
    return c;
}

// Random order (cpu_sa.cpp:134-139) in speculative windows of the RNG
// stream.  Each attempt draws its variable as rand % n and, when it needs one,
// its acceptance draw right after it.  Lane l takes stream position q + l as
// the variable draw of a possible attempt and q + l + 1 as that attempt's
// acceptance draw, and decides it against the delta energies at the start of
// the pass.  The attempts actually made form a chain: lane 0, then each
// chain lane's successor at l + 1, or l + 2 when l drew for its acceptance.
// A chain lane's decision stands unless an earlier accepted flip of the
// window touched its variable (flipped it or a neighbour of it); the window
// commits the chain up to the first such lane.  Touched variables are marked
// in a per-warp bitmap (`touch`, n bits, clear between passes).  Committed
// flips are pairwise distinct and non-adjacent, so their neighbour updates
// are applied together, equal targets summed in entry order.
template <bool GIBBS, bool REG, class DE>
__device__ __forceinline__ void sweep_random(const Prob &P, DE de,
                                             int8_t *sp, double *scratch,
                                             uint64_t *ring, RingState &rs,
                                             unsigned lane, uint32_t *touch) {
    const int n = P.n;
    const int D = REG ? P.regular_degree : 0;
    for (int b = 0; b < reload(P.pd->num_betas); ++b) {
        const double beta = __ldg(&reload(P.pd->betas)[b]);
        const double thr = __ldg(&reload(P.pd->thresholds)[b]);
        for (int sw = 0; sw < reload(P.pd->sweeps_per_beta); ++sw) {
            SweepCount cnt;
            int rem = n;  // attempts left in this sweep
            while (rem > 0) {
                ring_refill(ring, rs, lane);
                const uint64_t rv = ring[(rs.q + lane) & (kRing - 1)];
                const int var = (int)(rv % (uint64_t)n);  // cpu_sa.cpp:135-136
                const double d = de.get(var);
                const bool cons = !(d >= thr);            // cpu_sa.cpp:140
                const bool need = GIBBS ? cons : (cons && !(d <= 0.0));
                const unsigned N = __ballot_sync(kFull, need);
                // Chain lanes: l is on the chain unless l - 1 is a chain lane
                // that drew.  Inside a run of drawing lanes starting at a, the
                // chain takes a, a + 2, ...; elsewhere every lane.
                bool on = true;
                if (lane > 0 && ((N >> (lane - 1)) & 1u)) {
                    const unsigned starts = N & ~(N << 1);
                    const unsigned below = starts & ((2u << (lane - 1)) - 1u);
                    const int a = 31 - __clz(below);
                    on = (((int)lane - a) & 1) == 0;
                }
                unsigned C = __ballot_sync(kFull, on);
                if (__popc(C) > rem) {  // the sweep ends inside the window
                    unsigned t = C;
                    for (int i = 0; i < rem; ++i) t &= t - 1u;
                    C &= ~t;
                }
                const bool chain = (C >> lane) & 1u;
                bool acc = false, near = false;
                if (chain) {
                    acc = GIBBS ? false : cons;  // Metropolis: d <= 0 accepts
                    if (need) {
                        const uint64_t r = ring[(rs.q + lane + 1u) & (kRing - 1)];
                        const int x = decide<GIBBS>(d, beta, r);
                        acc = (x & 1) != 0;
                        near = (x & 2) != 0;
                    }
                }
                const unsigned A = __ballot_sync(kFull, acc);
                const int c = random_commit(P, D, touch, var, chain, A, lane);
                const unsigned cm = C & (c >= 32 ? kFull : ((1u << c) - 1u));
                const int last = 31 - __clz(cm);  // lane 0 is always committed
                rs.q += (uint32_t)(last + 1) + ((N >> last) & 1u);
                rem -= __popc(cm);
                const unsigned fm = A & cm;
                cnt.pass((unsigned)__popc(fm), (unsigned)__popc(__ballot_sync(kFull, near) & cm));
                if (fm) {
                    const int s_old = (int)sp[var];
                    const uint2 vi = D ? make_uint2((uint32_t)var * (uint32_t)D, (uint32_t)D)
                                       : __ldg(&P.vinfo[var]);
                    __syncwarp();
                    apply_flips<REG>(P, de, sp, scratch, fm, var, (int)vi.x, (int)(vi.y & kDegMask),
                                s_old, true, lane);
                }
            }
            cnt.flush(ring, lane);
        }
    }
}

// Adds the terms of lanes 0 to cnt - 1 to e, in lane order.
__device__ __forceinline__ double add_terms(double e, double t, int cnt, double *buf,
                                            unsigned lane) {
    if (buf) {
        buf[lane] = t;
        __syncwarp();
        if (cnt == 32) {
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const double2 x = *reinterpret_cast<const double2 *>(buf + j);
                e = __dadd_rn(__dadd_rn(e, x.x), x.y);
            }
        } else {
            for (int j = 0; j < cnt; ++j) e = __dadd_rn(e, buf[j]);
        }
        __syncwarp();
    } else {
        for (int j = 0; j < cnt; ++j) e = __dadd_rn(e, __shfl_sync(kFull, t, j));
    }
    return e;
}

// cpu_sa.cpp:210-227.  Terms are formed lane-parallel (each an exact
// rounding of the same operands); the running sum is strictly sequential.
// The sum's chain of n + m additions is the bound, so everything else is kept
// off it: the terms go through `buf` (32 doubles of shared memory, or null:
// shuffles, two per term), from where all lanes read them without waiting for
// the sum, and the next 32 couplers are loaded before the present ones are
// added.
// Measured against shuffles and loads in place (one B200, kernel time): descent,
// 8192 samples of n = 2048, 3.92 -> 3.53 ms; n = 4000, 3552 reads x 16 sweeps,
// 8.03 -> 7.67; n = 20011, 1023 reads x 48 sweeps, 73.0 -> 71.2; lattice L = 16,
// 1000 reads x 20 sweeps, 6.10 -> 5.93 (with the initial fields' lists read four
// entries at a time, load_state).
__device__ __forceinline__ double state_energy(const ProblemDev *PD, const int8_t *sp,
                                               double *buf, unsigned lane) {
    const int n = PD->n;
    const int64_t m = PD->m;
    const double *__restrict__ h = PD->h;
    const int32_t *__restrict__ cu = PD->cu;
    const int32_t *__restrict__ cv = PD->cv;
    const double *__restrict__ cw = PD->cw;
    double e = 0.0;
    for (int base = 0; base < n; base += 32) {
        const int v = base + (int)lane;
        const double t = v < n ? __dmul_rn((double)(int)sp[v], __ldg(&h[v])) : 0.0;
        e = add_terms(e, t, min(32, n - base), buf, lane);
    }
    int u = 0, v = 0;
    double w = 0.0;
    auto load = [&](int64_t c) {
        if (c < m) {
            u = __ldg(&cu[c]);
            v = __ldg(&cv[c]);
            w = __ldg(&cw[c]);
        }
    };
    load(lane);
    for (int64_t base = 0; base < m; base += 32) {
        // Lanes past the last coupler form a term that is not added.
        const double t = __dmul_rn(__dmul_rn((double)(int)sp[u], w), (double)(int)sp[v]);
        load(base + 32 + lane);
        e = add_terms(e, t, (int)min((int64_t)32, m - base), buf, lane);
    }
    return e;
}

template <bool GIBBS, bool RANDOM_ORDER, bool RESOLVE, bool REG, int STAGE>
__device__ __forceinline__ void anneal_read(const ProblemDev *PD, const int8_t *src,
                                            int8_t *dst, double *energy_out,
                                            double *de, int8_t *sp,
                                            double *scratch, uint64_t *ring,
                                            RingState &rs, unsigned lane, uint32_t *touch,
                                            double *band, int band_cap) {
    const bool pm1 = load_state(PD, src, de, sp, lane);
    {
        const Prob P = load_prob(PD);
        if constexpr (RANDOM_ORDER) {
            static_assert(STAGE != kStageBand, "the band follows a sequential window");
            typename DeFor<STAGE>::T acc;
            acc.p = de;
            sweep_random<GIBBS, REG>(P, acc, sp, scratch, ring, rs, lane, touch);
        } else {
            // A problem whose band does not fit the launch's ring keeps all of
            // its delta energies in the global slot.
            const int bw = (STAGE == kStageBand && PD->band_w > 0 && PD->band_w <= band_cap)
                               ? PD->band_w
                               : 0;
            if (RESOLVE && pm1)
                sweep_resolved<GIBBS, STAGE, REG>(P, de, sp, scratch, ring, rs, lane, band, bw,
                                             PD->band_b);
            else
                sweep_sequential<GIBBS, STAGE, REG>(P, de, sp, scratch, ring, rs, lane, band, bw,
                                               PD->band_b);
        }
    }
    __syncwarp();
    const double e = state_energy(PD, sp, scratch, lane);
    const int n = PD->n;
    for (int v = lane; v < n; v += 32) dst[v] = sp[v];
    if (lane == 0) *energy_out = e;
    __syncwarp();
}

}  // namespace b200sa
