// Simulated annealing of small problems with the state in registers.
// Included by sa_launch.cu; arithmetic as in sa_kernel.cuh.
//
// One warp per read.  Lane l owns the delta energies and spins of variables l,
// l + 32, ... (K of them), and the couplings are read from a dense matrix.  A
// flip is applied at once, in the reference's order, by every lane to its own
// variables (cpu_sa.cpp:168-191): d_x += ((int8)(4 s_j) J_jx) s_x, then the
// flipped variable's spin and delta energy are negated.  (Where x is not a
// neighbour J_jx is 0 and the addition leaves d_x as it was, but for the sign
// of a zero, which no decision sees.)  Nothing is deferred, so any spin values
// are handled; problems whose lists name a target twice are not (they keep the
// general path).
//
// What bounds it is the chain from one flip to the next decision: coupling
// load, a double product and sum, the acceptance bound in single precision, two
// votes (about 380 cycles with one read on an SM; 70 to 120 instructions).  The
// logarithms of a window's draws are taken beforehand, side by side, so that
// chain holds no conversion of a random number and no load of one.  Measured
// against the general path (delta energies and spins in shared memory, every
// round of a window reading its draws anew): dense n = 100, 1000 reads x 1000
// sweeps 9.6 -> 5.0 ms, random order 41.6 -> 11.1; K16 Gibbs, 4096 reads x 2000
// sweeps 13.6 -> 4.0; n = 300, 200 sweeps 20.2 -> 3.9, random order 28.6 -> 6.3;
// one read of K16 3.8 -> 1.7.
#pragma once
#include "sa_kernel.cuh"

namespace b200sa {

// The state of one read.  PM1: every spin is +1 or -1, kept as a sign bit; a
// contribution ((int8)(4 s_j) J) s_x is then J times +4 or -4, exactly.
template <bool PM1, int K>
struct DenseState;

template <int K>
struct DenseState<true, K> {
    double d[K];      // delta energies of variables lane + 32 i
    uint32_t neg[K];  // spins: 0 or the sign bit
    const double *w;  // coupling matrix, this lane's column
    int ld;           // row length (a multiple of 32)
    using Spin = uint32_t;

    static __device__ __forceinline__ uint32_t pack(int s) { return s < 0 ? 0x80000000u : 0u; }
    static __device__ __forceinline__ int unpack(uint32_t x) { return x ? -1 : 1; }
    static __device__ __forceinline__ uint32_t negated(uint32_t x) { return x ^ 0x80000000u; }
    // A flip's factor (cpu_sa.cpp:172), and its contribution to a variable of
    // spin x through coupling J.
    static __device__ __forceinline__ uint32_t factor(uint32_t x) { return x; }
    static __device__ __forceinline__ double term(uint32_t f, double J, uint32_t x) {
        return __dmul_rn(J, __hiloint2double((int)(0x40100000u ^ f ^ x), 0));
    }
    __device__ __forceinline__ uint32_t spin(int i) const { return neg[i]; }
    __device__ __forceinline__ void set_spin(int i, uint32_t x) { neg[i] = x; }
};

template <int K>
struct DenseState<false, K> {
    double d[K];
    int s[K];
    const double *w;
    int ld;
    using Spin = int;

    static __device__ __forceinline__ int pack(int s) { return s; }
    static __device__ __forceinline__ int unpack(int x) { return x; }
    static __device__ __forceinline__ int negated(int x) { return (int)(int8_t)(-x); }
    static __device__ __forceinline__ int factor(int x) { return (int)(int8_t)(4 * x); }
    static __device__ __forceinline__ double term(int f, double J, int x) {
        return __dmul_rn(__dmul_rn((double)f, J), (double)x);
    }
    __device__ __forceinline__ int spin(int i) const { return s[i]; }
    __device__ __forceinline__ void set_spin(int i, int x) { s[i] = x; }
};

// The contributions of a flip of variable v with factor f to every lane's
// variables (cpu_sa.cpp:172-185).  Slots past the end of the row read what
// follows it in the arena, into delta energies nothing looks at.
template <class STATE, int K>
__device__ __forceinline__ void dense_push(STATE &S, int v, typename STATE::Spin f) {
    const double *row = S.w + (size_t)v * (size_t)S.ld;
    double J[K];
#pragma unroll
    for (int i = 0; i < K; ++i) J[i] = __ldg(row + 32 * i);
#pragma unroll
    for (int i = 0; i < K; ++i) S.d[i] = __dadd_rn(S.d[i], STATE::term(f, J[i], S.spin(i)));
}

// One sweep in sequential order: windows of 32 variables, window w being slot w
// of every lane, whose delta energy d and spin s are taken out for the window
// and put back after it.  All lanes decide; accepted flips are applied one by
// one, and as soon as one of them touches a later lane of the window the lanes
// after it decide again (their draws placed after those before them).
template <bool GIBBS, bool PM1, int K>
__device__ __forceinline__ void dense_sweep_sequential(DenseState<PM1, K> &S, int n, double beta,
                                                       double thr, uint64_t *ring, RingState &rs,
                                                       unsigned lane, SweepCount &cnt) {
    using State = DenseState<PM1, K>;
    using Spin = typename State::Spin;
    const unsigned lt_mask = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7f800000);
    const float scale = Choice<GIBBS>::scale(beta);
    // (Unrolled only while the copies of the body stay small.)
#pragma unroll(K <= 4 ? K : 1)
    for (int w = 0; w < K; ++w) {
        const int L = n - 32 * w;
        if (L <= 0) break;
        const bool act = (int)lane < L;
        double d = 0.0;
        Spin s = 0;
#pragma unroll
        for (int i = 0; i < K; ++i)
            if (i == w) d = S.d[i], s = S.spin(i);
        Choice<GIBBS> ch;
        ch.look(d, scale, thr, act);
        unsigned nm = __ballot_sync(kFull, ch.need);
        unsigned flips = 0u, ties = 0u;
        // (A bound of NaN counts as a decision to be made.)
        if (__any_sync(kFull, !(ch.t == -inf))) {
            ring_refill(ring, rs, lane);
            const float y = draw_log2(ring[(rs.q + lane) & (kRing - 1)]);
            int c = 0;  // lanes below c are committed
            for (;;) {
                const int at = __popc(nm & lt_mask);
                const float gap = ch.t - __shfl_sync(kFull, y, at);
                unsigned am = __ballot_sync(kFull, gap > kBand);
                if (__any_sync(kFull, !(fabsf(gap) > kBand))) {  // inside the band
                    int x = 0;
                    if ((int)lane >= c && !(fabsf(gap) > kBand))
                        x = ch.exact(d, beta, ring[(rs.q + (uint32_t)at) & (kRing - 1)]);
                    am |= __ballot_sync(kFull, (x & 1) != 0);
                    ties |= __ballot_sync(kFull, (x & 2) != 0);
                }
                bool again = false;
                while (am) {
                    const int j = __ffs(am) - 1;
                    am &= am - 1u;
                    c = j + 1;
                    ++flips;
                    const Spin f = __shfl_sync(kFull, State::factor(s), j);
                    const double J =
                        __ldg(S.w + (size_t)(32 * w + j) * (size_t)S.ld + (size_t)(32 * w));
                    dense_push<State, K>(S, 32 * w + j, f);
                    d = __dadd_rn(d, State::term(f, J, s));
                    if ((int)lane == j) {  // cpu_sa.cpp:189-190
                        s = State::negated(s);
                        d = -d;
                    }
                    if (__any_sync(kFull, (int)lane > j && J != 0.0)) {
                        again = true;
                        break;
                    }
                }
                if (!again) break;
                // A tie of a lane that decides anew is no longer one.
                ties &= (1u << (c - 1)) | ((1u << (c - 1)) - 1u);
                Choice<GIBBS> next;
                next.look(d, scale, thr, act);
                const bool mine = (int)lane >= c;
                ch.t = mine ? next.t : -inf;  // committed lanes decide no more
                ch.need = mine ? next.need : ch.need;
                nm = __ballot_sync(kFull, ch.need);
            }
            rs.q += (uint32_t)__popc(nm);
#pragma unroll
            for (int i = 0; i < K; ++i)
                if (i == w) S.d[i] = d, S.set_spin(i, s);
        }
        cnt.pass(flips, (unsigned)__popc(ties));
    }
}

// One sweep in random order: windows of 32 stream positions (see
// sweep_random).  An accepted flip is applied to the owners' variables and to
// the copies that the later attempts of the window hold, and those it touches
// decide again, so a window always commits whole.
template <bool GIBBS, bool PM1, int K>
__device__ __forceinline__ void dense_sweep_random(DenseState<PM1, K> &S, int n, double beta,
                                                   double thr, uint64_t magic, uint64_t *ring,
                                                   RingState &rs, unsigned lane,
                                                   SweepCount &cnt) {
    using State = DenseState<PM1, K>;
    using Spin = typename State::Spin;
    const double *matrix = S.w - lane;
    const float scale = Choice<GIBBS>::scale(beta);
    for (int rem = n; rem > 0;) {
        ring_refill(ring, rs, lane);
        const int var = mod_n(ring[(rs.q + lane) & (kRing - 1)], (uint32_t)n, magic);
        const float y = draw_log2(ring[(rs.q + lane + 1u) & (kRing - 1)]);
        double d = 0.0;
        Spin s = 0;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            const double di = __shfl_sync(kFull, S.d[i], var & 31);
            const Spin si = __shfl_sync(kFull, S.spin(i), var & 31);
            if (var >> 5 == i) d = di, s = si;
        }
        Choice<GIBBS> ch;
        ch.look(d, scale, thr, true);
        unsigned flips = 0u, ties = 0u, live = kFull, C, N;
        for (;;) {
            N = __ballot_sync(kFull, ch.need);
            bool on = true;  // chain lanes, see sweep_random
            if (lane > 0 && ((N >> (lane - 1)) & 1u)) {
                const unsigned below = (N & ~(N << 1)) & ((2u << (lane - 1)) - 1u);
                on = (((int)lane - (31 - __clz(below))) & 1) == 0;
            }
            C = __ballot_sync(kFull, on);
            if (__popc(C) > rem) {
                unsigned t = C;
                for (int i = 0; i < rem; ++i) t &= t - 1u;
                C &= ~t;
            }
            const float gap = ch.t - y;
            unsigned am = __ballot_sync(kFull, gap > kBand) & C & live;
            if (__ballot_sync(kFull, !(fabsf(gap) > kBand)) & C & live) {  // inside the band
                int x = 0;
                if (((C & live) >> lane & 1u) && !(fabsf(gap) > kBand))
                    x = ch.exact(d, beta, ring[(rs.q + lane + 1u) & (kRing - 1)]);
                am |= __ballot_sync(kFull, (x & 1) != 0);
                ties |= __ballot_sync(kFull, (x & 2) != 0);
            }
            bool again = false;
            while (am) {
                const int j = __ffs(am) - 1;
                am &= am - 1u;
                flips |= 1u << j;
                live = (kFull - 1u) << j;
                const int vj = __shfl_sync(kFull, var, j);
                const Spin f = __shfl_sync(kFull, State::factor(s), j);
                const double J = __ldg(matrix + (size_t)vj * (size_t)S.ld + var);
                dense_push<State, K>(S, vj, f);
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    if (vj == (int)lane + 32 * i) {  // cpu_sa.cpp:189-190
                        S.set_spin(i, State::negated(S.spin(i)));
                        S.d[i] = -S.d[i];
                    }
                }
                if ((live >> lane) & 1u) {
                    d = __dadd_rn(d, State::term(f, J, s));
                    if (var == vj) {
                        s = State::negated(s);
                        d = -d;
                    }
                }
                if (__ballot_sync(kFull, J != 0.0 || var == vj) & live) {
                    again = true;
                    break;
                }
            }
            if (!again) break;
            ties &= ~live;
            Choice<GIBBS> next;
            next.look(d, scale, thr, true);
            if ((live >> lane) & 1u) ch = next;
        }
        const int last = 31 - __clz(C);  // lane 0 is always on the chain
        rs.q += (uint32_t)(last + 1) + ((N >> last) & 1u);
        rem -= __popc(C);
        cnt.pass((unsigned)__popc(flips), (unsigned)__popc(ties));
    }
}

template <bool GIBBS, bool RANDOM_ORDER, bool PM1, int K>
__device__ __forceinline__ void dense_anneal(const ProblemDev *PD, const int8_t *src, int8_t *sp,
                                             uint64_t *ring, RingState &rs, unsigned lane) {
    using State = DenseState<PM1, K>;
    const int n = PD->n;
    State S;
    S.ld = dense_ld(n);
    S.w = PD->dense_w + lane;
#pragma unroll
    for (int i = 0; i < K; ++i) {  // cpu_sa.cpp:54-74
        const int v = (int)lane + 32 * i;
        S.d[i] = 0.0;
        S.set_spin(i, 0);
        if (v < n) {
            const int x = (int)src[v];
            const uint2 vi = __ldg(&PD->vinfo[v]);
            double f = __ldg(&PD->h[v]);
            for (unsigned e = vi.x; e < vi.x + (vi.y & kDegMask); ++e)
                f = __dadd_rn(f, __dmul_rn((double)(int)src[__ldg(&PD->col[e])], __ldg(&PD->w[e])));
            S.d[i] = __dmul_rn((double)(-2 * x), f);
            S.set_spin(i, State::pack(x));
        }
    }
    const uint64_t magic = ~0ull / (uint64_t)n;
    const int num_betas = PD->num_betas, sweeps = PD->sweeps_per_beta;
    for (int b = 0; b < num_betas; ++b) {
        const double beta = __ldg(&PD->betas[b]);
        const double thr = __ldg(&PD->thresholds[b]);
        for (int sw = 0; sw < sweeps; ++sw) {
            SweepCount cnt;
            if constexpr (RANDOM_ORDER)
                dense_sweep_random<GIBBS, PM1, K>(S, n, beta, thr, magic, ring, rs, lane, cnt);
            else
                dense_sweep_sequential<GIBBS, PM1, K>(S, n, beta, thr, ring, rs, lane, cnt);
            cnt.flush(ring, lane);
        }
    }
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int v = (int)lane + 32 * i;
        if (v < n) sp[v] = (int8_t)State::unpack(S.spin(i));
    }
}

// One read.  `scratch` holds the final spins for the energy.
template <bool GIBBS, bool RANDOM_ORDER, int K>
__device__ __forceinline__ void dense_anneal_read(const ProblemDev *PD, const int8_t *src,
                                                  int8_t *dst, double *energy_out,
                                                  double *scratch, uint64_t *ring, RingState &rs,
                                                  unsigned lane) {
    const int n = PD->n;
    int8_t *sp = reinterpret_cast<int8_t *>(scratch);
    static_assert(32 * K <= kScratchHotBytes, "the spins fit the scratch");
    bool pm1 = true;
    for (int v = (int)lane; v < n; v += 32) pm1 = pm1 && (src[v] == 1 || src[v] == -1);
    if (__all_sync(kFull, pm1))
        dense_anneal<GIBBS, RANDOM_ORDER, true, K>(PD, src, sp, ring, rs, lane);
    else
        dense_anneal<GIBBS, RANDOM_ORDER, false, K>(PD, src, sp, ring, rs, lane);
    __syncwarp();
    for (int v = (int)lane; v < n; v += 32) dst[v] = sp[v];
    __syncwarp();
    const double e = state_energy(PD, sp, nullptr, lane);
    if (lane == 0) *energy_out = e;
    __syncwarp();
}

}  // namespace b200sa
