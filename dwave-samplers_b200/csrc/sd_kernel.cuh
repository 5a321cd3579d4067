// Steepest descent kernel (included by sa_launch.cu, next to the annealing
// kernels whose helpers it shares).
// The drop-in for the reference's
// steepest_gradient_descent (dwave/samplers/greedy/src/descent.cpp:315-405),
// the step usually run after annealing to take every sample to a local
// minimum.  One warp per sample.
//
// Arithmetic follows descent.cpp operation for operation:
//   flip energy (descent.cpp:41-60) = -2*s * (h + sum s_nb*J, adjacency order),
//     the same expression as the annealer's delta energy (load_state);
//   selection (descent.cpp:149-156, 234-238): the least flip energy, ties to
//     the lower index, and only a negative one is taken;
//   linear-search solver (:161-182): s *= -1, fe[v] *= -1, then every list
//     entry fe[nb] -= ((4*s_new) * J) * s_nb in list order;
//   ordered-set solver (:255-285, large_sparse_opt): every list entry
//     fe[nb] += ((4*s_old) * J) * s_nb in list order, then s *= -1 and fe[v]
//     set to minus its value before the list loop;
//   state energy (:75-93) as state_energy.
// Descent stops when no flip energy is negative, or after max_steps steps:
// with a self-loop of positive weight (or spins other than +-1) a variable
// can flip back and forth for ever (the reference never returns then); here
// the sample stops at max_steps and the call reports B200SA_ETIMEOUT.
#pragma once
#include "sa_kernel.cuh"

namespace b200sa {
// Finding the least flip energy bounds a step.  Variables form groups of 32
// consecutive ones, and each group's least negative-energy key and its variable
// are kept: a step looks at n / 32 groups, one to a lane and round, and scans
// again only the groups where it may have changed, that of the flipped variable
// and a few of its neighbours'.  (Scanning all n, or from n = 4096 on keeping
// the minimum of each lane's n / 32 variables, took 7.0 ms for 8192 samples of n
// = 2048, 6-regular; this takes 3.9 ms.  What is left is the latency of a step,
// about 1700 cycles: the list from L2, three reductions each for the least
// group and for the flipped group.  Fetching the list of the next group minimum
// ahead gained nothing: its reductions cost what it saved.)  With few groups, or
// lists so long that a flip leaves few groups as they were, a step looks at all
// variables instead (FLAT, sd_flat).
//
// A key orders negative energies (more negative is smaller); every other value,
// NaN included, is kSdNone, never chosen.
constexpr unsigned long long kSdNone = ~0ull;
__device__ __forceinline__ unsigned long long sd_key(double e) {
    return e < 0.0 ? ~(unsigned long long)__double_as_longlong(e) : kSdNone;
}

// The least key of the warp, and the least `v` among the lanes that hold it.
__device__ __forceinline__ void warp_least(unsigned long long &key, unsigned &v) {
    const unsigned hi = __reduce_min_sync(kFull, (unsigned)(key >> 32));
    const bool a = (unsigned)(key >> 32) == hi;
    const unsigned lo = __reduce_min_sync(kFull, a ? (unsigned)key : ~0u);
    v = __reduce_min_sync(kFull, a && (unsigned)key == lo ? v : ~0u);
    key = ((unsigned long long)hi << 32) | lo;
}

// A sample's group minima: keys, and the variable's place in its group.
struct SdGroups {
    unsigned long long *key;
    uint8_t *at;

    __device__ __forceinline__ void scan(const double *fe, int g, int n, unsigned lane) const {
        const int v = 32 * g + (int)lane;
        unsigned long long k = v < n ? sd_key(fe[v]) : kSdNone;
        unsigned at_lane = lane;
        warp_least(k, at_lane);
        if (lane == 0) {
            key[g] = k;
            at[g] = (uint8_t)at_lane;
        }
    }
};

template <bool SPARSE, bool SMEM, bool FLAT>
__global__ void __launch_bounds__(kMaxThreadsPerCta, 1)
    sd_warp_kernel(SdArgs A, int warps_per_cta, int region_bytes) {
    extern __shared__ __align__(16) uint8_t smem[];
    const unsigned lane = threadIdx.x & 31u;
    const int wid = (int)(threadIdx.x >> 5);
    uint8_t *region = smem + A.table_bytes + (size_t)wid * (size_t)region_bytes;
    double *scratch = reinterpret_cast<double *>(region);
    const int64_t gw = (int64_t)blockIdx.x * warps_per_cta + wid;
    const ProblemDev *PD = A.problem;
    const Prob P = load_prob(PD);
    const int n = P.n;
    // A step's list start is computed (equal lists) or read from a table in
    // shared memory (SMEM), one trip to L2 less in its chain.
    const int D = P.regular_degree;
    uint32_t *starts = reinterpret_cast<uint32_t *>(smem);
    if (SMEM && A.table_bytes) {
        for (int v = (int)threadIdx.x; v <= n; v += (int)blockDim.x)
            starts[v] = v < n ? __ldg(&P.vinfo[v]).x : 2u * (uint32_t)PD->m;
        __syncthreads();
    }
    auto list = [&](int v) {  // start and degree
        if (D) return make_uint2((uint32_t)v * (uint32_t)D, (uint32_t)D);
        if (SMEM) return make_uint2(starts[v], starts[v + 1] - starts[v]);
        const uint2 vi = __ldg(&P.vinfo[v]);
        return make_uint2(vi.x, vi.y & kDegMask);
    };
    const int groups = (n + 31) / 32;
    double *fe;
    int8_t *sp;
    SdGroups G;
    if (SMEM) {
        fe = reinterpret_cast<double *>(region + kSdScratchBytes);
        G.key = reinterpret_cast<unsigned long long *>(fe + n);
        sp = reinterpret_cast<int8_t *>(G.key + groups);
        G.at = reinterpret_cast<uint8_t *>(sp + n);
    } else {
        fe = A.scratch_fe + gw * A.scratch_stride;
        sp = A.scratch_s + gw * A.scratch_stride;
        G.key = A.scratch_key + gw * A.group_stride;
        G.at = A.scratch_at + gw * A.group_stride;
    }
    for (;;) {
        unsigned long long x = 0;
        if (lane == 0) x = atomicAdd(A.queue_head, 1ull);
        const int64_t it = (int64_t)__shfl_sync(kFull, x, 0);
        if (it >= A.num_items) break;
        const int r = (int)(A.items[it] & 0xffffffffll);
        const int64_t so = PD->state_offset + (int64_t)r * n;
        load_state(PD, A.states_in + so, fe, sp, lane);  // descent.cpp:41-60, 128-133
        for (int g = 0; !FLAT && g < groups; ++g) G.scan(fe, g, n, lane);
        __syncwarp();
        uint32_t steps = 0;
        bool capped = false;
        for (;;) {
            // descent.cpp:149-156 / 234-238: the least negative flip energy,
            // ties to the lowest index.
            unsigned long long bk = kSdNone;
            unsigned best = ~0u;
            if constexpr (FLAT) {
#pragma unroll 4
                for (int v = (int)lane; v < n; v += 32) {
                    const unsigned long long k = sd_key(fe[v]);
                    if (k < bk) {
                        bk = k;
                        best = (unsigned)v;
                    }
                }
            } else {
                for (int g = (int)lane; g < groups; g += 32) {
                    const unsigned long long k = G.key[g];
                    if (k < bk) {
                        bk = k;
                        best = 32u * (unsigned)g + G.at[g];
                    }
                }
            }
            warp_least(bk, best);
            if (bk == kSdNone) break;  // :159-161 / :244
            if (steps >= A.max_steps) {
                capped = true;
                break;
            }
            const int bv = (int)best;
            [[maybe_unused]] const double be = __longlong_as_double((long long)~bk);
            const uint2 vi = list(bv);
            const int start = (int)vi.x, deg = (int)vi.y;
            int col0 = 0;  // entry `lane`
            double w0 = 0.0;
            if ((int)lane < deg) {
                col0 = __ldg(&P.col[start + (int)lane]);
                w0 = __ldg(&P.w[start + (int)lane]);
            }
            const int s_old = (int)sp[bv];
            const int s_new = (int)(int8_t)(s_old * -1);
            __syncwarp();
            if (!SPARSE && lane == 0) {  // :168, :172
                sp[bv] = (int8_t)s_new;
                fe[bv] = __dmul_rn(fe[bv], -1.0);
            }
            __syncwarp();
            // List entries 32 at a time; equal targets within a round are
            // applied by their first lane in entry order.
            const bool dup = A.any_dup && (__ldg(&P.share[bv]) & 1u) != 0u;
            const double mult = (double)(4 * (SPARSE ? s_old : s_new));
            for (int base = 0; base < deg; base += 32) {
                const int k = base + (int)lane;
                const bool a = k < deg;
                int nb = -1 - (int)lane;
                double xk = 0.0;
                if (a) {
                    nb = base ? __ldg(&P.col[start + k]) : col0;
                    const double wk = base ? __ldg(&P.w[start + k]) : w0;
                    xk = __dmul_rn(__dmul_rn(mult, wk), (double)(int)sp[nb]);
                }
                const unsigned grp = dup ? __match_any_sync(kFull, nb) : (1u << lane);
                const bool alone = grp == (1u << lane);
                if (a && alone) fe[nb] = SPARSE ? __dadd_rn(fe[nb], xk) : __dsub_rn(fe[nb], xk);
                if (dup && __any_sync(kFull, a && !alone)) {  // warp-uniform
                    scratch[lane] = xk;
                    __syncwarp();
                    if (a && !alone && lane == (unsigned)(__ffs(grp) - 1)) {
                        double acc = fe[nb];
                        unsigned g = grp;
                        while (g) {
                            const int j = __ffs(g) - 1;
                            g &= g - 1;
                            acc = SPARSE ? __dadd_rn(acc, scratch[j]) : __dsub_rn(acc, scratch[j]);
                        }
                        fe[nb] = acc;
                    }
                }
                __syncwarp();
            }
            if (SPARSE && lane == 0) {  // :280, :283-285
                sp[bv] = (int8_t)s_new;
                fe[bv] = __dmul_rn(be, -1.0);
            }
            __syncwarp();
            ++steps;
            if (FLAT) continue;
            // Groups whose minimum may have changed: the flipped variable's,
            // and those where a neighbour was it or falls below it.
            G.scan(fe, bv >> 5, n, lane);
            __syncwarp();
            for (int base = 0; base < deg; base += 32) {
                const int k = base + (int)lane;
                bool stale = false;
                int g = -1;
                if (k < deg) {
                    const int x = base ? __ldg(&P.col[start + k]) : col0;
                    g = x >> 5;
                    const unsigned long long kx = sd_key(fe[x]), kg = G.key[g];
                    const int least = 32 * g + (int)G.at[g];
                    stale = x == least ? kx != kg : kx < kg || (kx == kg && x < least);
                }
                __syncwarp();
                for (unsigned m; (m = __ballot_sync(kFull, stale)) != 0u;) {
                    const int gj = __shfl_sync(kFull, g, __ffs(m) - 1);
                    G.scan(fe, gj, n, lane);
                    if (g == gj) stale = false;
                }
                __syncwarp();
            }
        }
        __syncwarp();
        const double e = state_energy(PD, sp, scratch, lane);  // descent.cpp:75-93
        for (int v = lane; v < n; v += 32) A.states_out[so + v] = sp[v];
        if (lane == 0) {
            A.energies[PD->read_offset + r] = e;
            A.steps[PD->read_offset + r] = steps;
            if (capped) atomicAdd(A.capped, 1ull);
        }
        __syncwarp();
    }
}

}  // namespace b200sa

