// Rotor-model annealing (the reference's SQA rotor Monte Carlo,
// dwave/samplers/sqa/src/cpu_rotormc.cpp) on the GPU.  Included by
// sa_launch.cu next to the annealing kernels.
//
// One warp per sample, the sample's state on chip.  A sample is one sequential
// chain of attempts, so what bounds it is the latency of a step of that chain;
// the warp takes many attempts per step speculatively, from the RNG ring of
// the annealing kernel:
//
// * Non-ergodic proposals (a reflection): windows of 32 variables as in
//   sweep_sequential / sweep_random.  A reflection keeps a delta energy per
//   variable, and an attempt's draws are the same as the annealer's.
// * Uniform and transverse-field proposals recompute the local field and draw
//   for every attempt, so the stream position of attempt i of a window depends
//   on how many of the attempts before it drew for their acceptance.  In
//   sequential order the 28 lanes (i, o) with o <= i < 7 decide attempt i at
//   every possible offset o at once, and a walk over seven bits picks the ones
//   made; the fields of 32 variables are added up lane-parallel beforehand and
//   stay valid up to the first neighbour of a changed variable.  In random
//   order each lane takes one stream position as the start of a possible
//   attempt, as in sweep_random.
//
// With one thread per sample (rmc_thread_kernel) an attempt of a chain takes 0.5
// to 3 microseconds, by where its state lies, whatever the number of samples up
// to about 20,000 of them.  Measured, n = 512 6-regular, 64 sweeps: 4096 samples
// of reflections 67.5 ms with one thread per sample, 5.3 ms with a warp; 32768
// samples (32 sweeps) 55.8 against 20.4 ms; 1000 samples of transverse-field
// proposals 44.8 against 5.8 ms.  With few variables or very many samples the
// thread is the faster one (n = 9, 262144 samples, 111 sweeps of reflections:
// 4.2 ms against 38.7, random order 6.2 against 109): rmc_thread_samples.
//
// Arithmetic follows cpu_rotormc.cpp operation for operation:
//   local field (:46-60)       h + cos(theta_nb) * J, adjacency order
//   non-ergodic delta (:130-139) field * (-2 * cos(theta))
//   burn-in (:141-143)         32 draws before the first sweep of every run
//   Metropolis / Gibbs (:167-196), uniform and transverse-field proposals
//   (:197-266), updates (:268-287), statistics (:289-293), energy (:310-326).
// cos / |sin| of the 256 angles come from the host (cpu_rotormc.cpp:377-383,
// the host libm), copied into shared memory.
#pragma once
#include "sa_kernel.cuh"

namespace b200sa {

// exp(x) * 2^64 > (double)r.  Bit 0: accept; bit 1: the draw lies within the
// cross-libm tie band.  Outside (-44.4, 0] the single-precision bounds do not
// hold; below it a nonzero draw is always rejected (exp(x) * 2^64 < 1).
__device__ __forceinline__ int rmc_metropolis(double x, uint64_t r) {
    if (x <= 0.0) {
        if (x > -44.4) {
            const int fast = metropolis_fast(x, r);
            if (fast >= 0) return fast;
        } else if (x < -45.0 && r != 0) {
            return 0;
        }
    }
    return metropolis_exact(-x, 1.0, r);
}

// 2^64 > (double)r * (1 + exp(z)), the same bits.
__device__ __forceinline__ int rmc_gibbs(double z, uint64_t r) {
    if (z < 44.4) {
        const int fast = gibbs_fast(z, r);
        if (fast >= 0) return fast;
    } else if (z > 45.0 && r != 0) {
        return 0;
    }
    return gibbs_exact(z, 1.0, r);
}

// What a warp works on.
template <class DE>
struct RmcWarp {
    Prob P;
    const RmcArgs *A;
    DE de;          // non-ergodic proposals: delta energies
    uint8_t *st;    // angles
    const double *cs, *sn;
    double *scratch;
    uint64_t *ring;
    uint32_t *touch;  // random order: bitmap, clear between windows
    unsigned lane;
    unsigned near;  // warp-uniform
};

template <class DE>
__device__ __forceinline__ double rmc_field(const RmcWarp<DE> &W, int var) {
    const uint2 vi = __ldg(&W.P.vinfo[var]);
    double e = __ldg(&W.A->h[var]);
    for (unsigned k = vi.x; k < vi.x + vi.y; ++k)
        e = __dadd_rn(e, __dmul_rn(W.cs[W.st[__ldg(&W.P.col[k])]], __ldg(&W.P.w[k])));
    return e;
}

// The committed reflections `fm` of a window: neighbour updates (:270-283),
// then each flip's own delta energy -d and angle.
template <bool REG, class DE>
__device__ __forceinline__ void rmc_reflect(RmcWarp<DE> &W, unsigned fm, int v, uint2 vi,
                                            uint8_t cur, double d, bool may_conflict) {
    const uint8_t prop = (uint8_t)(128 + cur);
    const double mult = __dmul_rn(2.0, __dsub_rn(W.cs[cur], W.cs[prop]));
    push_entries<REG>(W.P, W.de, [&](int x) { return W.cs[W.st[x]]; }, W.scratch, fm, v, (int)vi.x,
                 (int)vi.y, mult, may_conflict, W.lane);
    if ((fm >> W.lane) & 1u) {
        W.st[v] = prop;
        W.de.set(v, -d);
    }
    __syncwarp();
}

// One sweep of reflections in sequential order: speculative windows as in
// sweep_sequential (without its threshold: every uphill attempt draws).
template <bool GIBBS, class DE>
__device__ __forceinline__ void rmc_reflect_sequential(RmcWarp<DE> &W, RingState &rs,
                                                       double beta) {
    const Prob &P = W.P;
    const unsigned lane = W.lane;
    const unsigned lt_mask = (1u << lane) - 1u;
    for (int p = 0; p < P.n;) {
        ring_refill(W.ring, rs, lane);
        const int L = min(32, P.n - p);
        const int v = p + (int)lane;
        const bool act = (int)lane < L;
        double d = 0.0;
        int dist = (int)kDistCap;
        uint32_t shr = 0u;
        uint2 vi = make_uint2(0u, 0u);
        uint8_t cur = 0;
        if (act) {
            d = W.de.get(v);
            dist = __ldg(&P.dist[v]);
            shr = __ldg(&P.share[v]);
            vi = __ldg(&P.vinfo[v]);
            cur = W.st[v];
        }
        const bool need = act && (GIBBS || !(d <= 0.0));
        const unsigned nm = __ballot_sync(kFull, need);
        bool acc = act && !need, near = false;
        if (need) {
            const uint64_t r = W.ring[(rs.q + (uint32_t)__popc(nm & lt_mask)) & (kRing - 1)];
            const int x = GIBBS ? rmc_gibbs(__dmul_rn(d, beta), r)
                                : rmc_metropolis(__dmul_rn(-d, beta), r);
            acc = (x & 1) != 0;
            near = (x & 2) != 0;
        }
        const unsigned am = __ballot_sync(kFull, acc);
        const int c = min(__reduce_min_sync(kFull, acc ? (int)lane + dist : 32), L);
        const unsigned done = c >= 32 ? kFull : ((1u << c) - 1u);
        rs.q += (uint32_t)__popc(nm & done);
        W.near += (unsigned)__popc(__ballot_sync(kFull, near) & done);
        const unsigned fm = am & done;
        if (fm) {
            const unsigned later = lane < 31 ? fm >> (lane + 1) : 0u;
            const bool f = (fm >> lane) & 1u;
            const bool may_conflict =
                __any_sync(kFull, f && ((shr & 1u) || ((shr >> 1) & later)));
            if (P.regular_degree)
                rmc_reflect<true>(W, fm, v, vi, cur, d, may_conflict);
            else
                rmc_reflect<false>(W, fm, v, vi, cur, d, may_conflict);
        }
        p += c;
    }
}

// One sweep of reflections in random order: windows of the RNG stream as in
// sweep_random.
template <bool GIBBS, class DE>
__device__ __forceinline__ void rmc_reflect_random(RmcWarp<DE> &W, RingState &rs, double beta,
                                                   uint64_t magic) {
    const Prob &P = W.P;
    const unsigned lane = W.lane;
    for (int rem = P.n; rem > 0;) {
        ring_refill(W.ring, rs, lane);
        const int var = mod_n(W.ring[(rs.q + lane) & (kRing - 1)], (uint32_t)P.n, magic);
        const double d = W.de.get(var);
        const bool need = GIBBS || !(d <= 0.0);
        const unsigned N = __ballot_sync(kFull, need);
        bool on = true;  // chain lanes, see sweep_random
        if (lane > 0 && ((N >> (lane - 1)) & 1u)) {
            const unsigned below = (N & ~(N << 1)) & ((2u << (lane - 1)) - 1u);
            on = (((int)lane - (31 - __clz(below))) & 1) == 0;
        }
        unsigned C = __ballot_sync(kFull, on);
        if (__popc(C) > rem) {
            unsigned t = C;
            for (int i = 0; i < rem; ++i) t &= t - 1u;
            C &= ~t;
        }
        const bool chain = (C >> lane) & 1u;
        bool acc = chain && !need, near = false;
        if (chain && need) {
            const uint64_t r = W.ring[(rs.q + lane + 1u) & (kRing - 1)];
            const int x = GIBBS ? rmc_gibbs(__dmul_rn(d, beta), r)
                                : rmc_metropolis(__dmul_rn(-d, beta), r);
            acc = (x & 1) != 0;
            near = (x & 2) != 0;
        }
        const unsigned A = __ballot_sync(kFull, acc);
        const int c = random_commit(P, 0, W.touch, var, chain, A, lane);
        const unsigned cm = C & (c >= 32 ? kFull : ((1u << c) - 1u));
        const int last = 31 - __clz(cm);  // lane 0 is always committed
        rs.q += (uint32_t)(last + 1) + ((N >> last) & 1u);
        rem -= __popc(cm);
        W.near += (unsigned)__popc(__ballot_sync(kFull, near) & cm);
        const unsigned fm = A & cm;
        if (fm) {
            const uint2 vi = __ldg(&P.vinfo[var]);
            const uint8_t cur = W.st[var];
            __syncwarp();
            if (P.regular_degree)
                rmc_reflect<true>(W, fm, var, vi, cur, d, true);
            else
                rmc_reflect<false>(W, fm, var, vi, cur, d, true);
        }
    }
}

// A proposed angle and whether it is taken.
struct RmcStep {
    uint8_t prop;
    bool need, flip, near;
};

// The schedule step's proposal parameters (:208-213); `tf` false: uniform.
struct RmcProposal {
    bool tf;
    int osi;
    uint32_t span, two32;  // 2 osi + 1 (0: not below 2^16) and 2^32 mod it
    double p;      // probability of the outermost angles, as a threshold times 2^64
    double beta, beta_tf;
};

template <int PROPOSAL>
__device__ __forceinline__ RmcProposal rmc_proposal(double beta, double beta_tf) {
    RmcProposal q;
    q.beta = beta;
    q.beta_tf = beta_tf;
    const double rat = __ddiv_rn(beta_tf, beta);
    q.tf = PROPOSAL == 3 && !(rat >= 1);
    q.osi = 0;
    q.span = q.two32 = 0u;
    q.p = 0.0;
    if (q.tf) {
        q.osi = (int)__dsub_rn(__dmul_rn(rat, 128.0), 0.5);
        const double distc = __ddiv_rn((double)(q.osi * (q.osi + 1)), (double)(2 * q.osi + 1));
        q.p = __dmul_rn(__ddiv_rn(__dsub_rn(__dmul_rn(__ddiv_rn(rat, 2.0), 128.0), distc),
                                  __dsub_rn((double)(q.osi + 1), distc)),
                        kTwo64);
        if (q.osi >= 0 && q.osi < 32768) {
            q.span = (uint32_t)(2 * q.osi + 1);
            q.two32 = (0u - q.span) % q.span;
        }
    }
    return q;
}

// x % (uint64_t)(2 * osi + 1).
__device__ __forceinline__ uint64_t rmc_mod(const RmcProposal &q, uint64_t x) {
    if (q.span)
        return (((uint32_t)(x >> 32) % q.span) * q.two32 + (uint32_t)x % q.span) % q.span;
    return x % (uint64_t)(2 * q.osi + 1);
}

// The proposed angle (:197-233); r2 is the second draw of the transverse-field
// proposal.
__device__ __forceinline__ uint8_t rmc_angle(const RmcProposal &q, uint8_t cur, uint64_t r1,
                                             uint64_t r2) {
    if (!q.tf) return (uint8_t)(r1 % 256);
    const uint8_t pac = q.p > __ull2double_rn(r1)
                            ? (uint8_t)((uint64_t)(q.osi + 1) * (2 * (r2 % 2) - 1))
                            : (uint8_t)(rmc_mod(q, r2) - (uint64_t)q.osi);
    return (uint8_t)(cur + pac);
}

// The proposal's log acceptance ratio (:234-247) from the local field e, the
// transverse field t and the cosines and sines of both angles.
__device__ __forceinline__ double rmc_log_ratio(const RmcProposal &q, double e, double t,
                                                double cs1, double cs0, double sn1, double sn0) {
    return __dadd_rn(__dmul_rn(__dmul_rn(-q.beta, e), __dsub_rn(cs1, cs0)),
                     __dmul_rn(__dmul_rn(q.beta_tf, t), __dsub_rn(sn1, sn0)));
}

// One attempt (:197-266) on a variable of angle `cur`, local field `e` and
// transverse field `t`, its draws starting at stream position `pos`.
template <class DE>
__device__ __forceinline__ RmcStep rmc_attempt(const RmcWarp<DE> &W, const RmcProposal &q,
                                               uint8_t cur, double e, double t, uint32_t pos) {
    RmcStep s;
    const uint64_t r1 = W.ring[pos & (kRing - 1)];
    const uint64_t r2 = W.ring[(pos + 1u) & (kRing - 1)];
    s.prop = rmc_angle(q, cur, r1, r2);
    const double dlm = rmc_log_ratio(q, e, t, W.cs[s.prop], W.cs[cur], W.sn[s.prop], W.sn[cur]);
    s.need = !(dlm >= 0.0);
    s.flip = true;
    s.near = false;
    if (s.need) {
        const int x = rmc_metropolis(
            dlm, q.tf ? W.ring[(pos + 2u) & (kRing - 1)] : r2);
        s.flip = (x & 1) != 0;
        s.near = (x & 2) != 0;
    }
    return s;
}

// Attempts per step in sequential order: the triangle of 28 lanes.
constexpr int kRmcTri = 7;
__device__ __forceinline__ constexpr int rmc_tri(int i) { return i * (i + 1) / 2; }

// One sweep of uniform or transverse-field proposals in sequential order.
template <class DE>
__device__ __forceinline__ void rmc_angle_sequential(RmcWarp<DE> &W, RingState &rs,
                                                     const RmcProposal &q) {
    const Prob &P = W.P;
    const unsigned lane = W.lane;
    const uint32_t K = q.tf ? 2u : 1u;  // proposal draws of an attempt
    int i = 0;                          // this lane's attempt within a step
    while (i < kRmcTri - 1 && rmc_tri(i + 1) <= (int)lane) ++i;
    const int o = (int)lane - rmc_tri(i);  // acceptance draws assumed before it
    for (int p = 0; p < P.n;) {
        // Fields of the window, valid for the variables below `end`.
        const int v = p + (int)lane;
        double e_w = 0.0, t_w = 0.0;
        int dist_w = (int)kDistCap, cur_w = 0;
        if (v < P.n) {
            e_w = rmc_field(W, v);
            t_w = __ldg(&W.A->tf[v]);
            dist_w = __ldg(&P.dist[v]);
            cur_w = W.st[v];
        }
        __syncwarp();
        int end = min(32, P.n - p);
        for (int b = 0; b < end;) {
            ring_refill(W.ring, rs, lane);
            const int L = min(kRmcTri, end - b);
            const int src = min(b + i, 31);
            const double e = __shfl_sync(kFull, e_w, src);
            const double t = __shfl_sync(kFull, t_w, src);
            const int dist = __shfl_sync(kFull, dist_w, src);
            const int cur = __shfl_sync(kFull, cur_w, src);
            const bool act = (int)lane < rmc_tri(L);
            RmcStep s{};
            if (act)
                s = rmc_attempt(W, q, (uint8_t)cur, e, t, rs.q + K * (uint32_t)i + (uint32_t)o);
            const unsigned N = __ballot_sync(kFull, s.need);
            // The lanes of the attempts made: each one's offset is the number
            // of draws before it.
            unsigned made = 0u;
            int at = 0;
#pragma unroll
            for (int k = 0; k < kRmcTri; ++k) {
                const int x = rmc_tri(k) + at;
                made |= 1u << x;
                at += (int)((N >> x) & 1u);
            }
            const bool mine = act && ((made >> lane) & 1u);
            const bool flip = mine && s.flip;
            // A changed variable ends the window at its nearest later neighbour.
            end = min(end, (int)__reduce_min_sync(kFull, flip ? b + i + dist : 64));
            const int c = min(L, end - b);  // > 0: dist >= 1
            const unsigned cm = made & ((1u << rmc_tri(c)) - 1u);
            rs.q += K * (uint32_t)c + (uint32_t)__popc(N & cm);
            W.near += (unsigned)__popc(__ballot_sync(kFull, mine && s.near) & cm);
            if (flip && i < c) W.st[p + b + i] = s.prop;
            b += c;
        }
        __syncwarp();
        p += end;
    }
}

// One sweep of uniform or transverse-field proposals in random order.
template <class DE>
__device__ __forceinline__ void rmc_angle_random(RmcWarp<DE> &W, RingState &rs,
                                                 const RmcProposal &q, uint64_t magic) {
    const Prob &P = W.P;
    const unsigned lane = W.lane;
    const int K = q.tf ? 3 : 2;  // draws of an attempt before its acceptance draw
    for (int rem = P.n; rem > 0;) {
        ring_refill(W.ring, rs, lane);
        const int var = mod_n(W.ring[(rs.q + lane) & (kRing - 1)], (uint32_t)P.n, magic);
        const uint8_t cur = W.st[var];
        const RmcStep s = rmc_attempt(W, q, cur, rmc_field(W, var), __ldg(&W.A->tf[var]),
                                      rs.q + lane + 1u);
        const unsigned N = __ballot_sync(kFull, s.need);
        unsigned C = 0u;  // the attempts made, in stream order
        int x = 0;
        for (int k = 0; x < 32 && k < rem; ++k) {
            C |= 1u << x;
            x += K + (int)((N >> x) & 1u);
        }
        const bool chain = (C >> lane) & 1u;
        const unsigned F = __ballot_sync(kFull, chain && s.flip);
        const int c = random_commit(P, 0, W.touch, var, chain, F, lane);
        const unsigned cm = C & (c >= 32 ? kFull : ((1u << c) - 1u));
        const int last = 31 - __clz(cm);  // lane 0 is always committed
        rs.q += (uint32_t)(last + K) + ((N >> last) & 1u);
        rem -= __popc(cm);
        W.near += (unsigned)__popc(__ballot_sync(kFull, s.near) & cm);
        if ((F & cm) >> lane & 1u) W.st[var] = s.prop;
        __syncwarp();
    }
}

// A warp mostly waits on its own chain, so residency counts: three CTAs of 256
// threads per SM (80 registers), and four (64) where the body fits them, which
// is sequential reflections on chip (4096 samples, n = 512, 64 sweeps: 7.2 ms
// at three, 5.3 at four; random order 21.0 at three, 28.1 at four).
template <bool RANDOM_ORDER, int PROPOSAL, int STAGE>
constexpr int kRmcCtas = !RANDOM_ORDER && PROPOSAL <= 1 && STAGE == kStageShared ? 4 : 3;

template <bool RANDOM_ORDER, int PROPOSAL, int STAGE>
__global__ void
__launch_bounds__(32 * kRmcMaxWarps, (kRmcCtas<RANDOM_ORDER, PROPOSAL, STAGE>))
    rmc_kernel(RmcArgs A) {
    extern __shared__ __align__(16) uint8_t smem[];
    double *cs = reinterpret_cast<double *>(smem);
    double *sn = cs + 256;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        cs[i] = A.cos_table[i];
        sn[i] = A.sin_table[i];
    }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    const int wid = (int)(threadIdx.x >> 5);
    const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + wid;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    if (A.shared_stream && gw != 0) return;
    uint8_t *region = smem + kRmcTableBytes + (size_t)wid * (size_t)A.region_bytes;
    RmcWarp<typename DeFor<STAGE>::T> W;
    W.ring = reinterpret_cast<uint64_t *>(region);
    W.scratch = reinterpret_cast<double *>(region + kRing * sizeof(uint64_t));
    uint8_t *state = region + kRing * sizeof(uint64_t) + kScratchBytes;
    if (A.touch) {
        W.touch = A.touch + gw * (A.touch_bytes / 4);
    } else {
        W.touch = reinterpret_cast<uint32_t *>(state);
        state += A.touch_bytes;
    }
    if constexpr (STAGE == kStageShared) {
        W.de.p = reinterpret_cast<double *>(state);
        W.st = state + (((size_t)A.n * sizeof(double) + 15) & ~size_t(15));
    } else {
        W.de.p = PROPOSAL <= 1 ? A.de + gw * A.slot_stride : nullptr;
        W.st = STAGE == kStageSpins ? state : A.states + gw * A.slot_stride;
    }
    W.A = &A;
    W.cs = cs;
    W.sn = sn;
    W.lane = lane;
    W.near = 0;
    const int n = A.n;
    Prob &P = W.P;
    P = Prob{};
    P.n = n;
    P.vinfo = A.vinfo;
    P.col = A.col;
    P.w = A.w;
    P.dist = A.dist;
    P.share = A.share;
    P.regular_degree = A.regular_degree;
    P.regular_magic = A.regular_magic;
    if (RANDOM_ORDER) {
        for (int i = (int)lane; i < A.touch_bytes / 4; i += 32) W.touch[i] = 0u;
        __syncwarp();
    }
    const uint64_t magic = ~0ull / (uint64_t)n;
    const int points = A.interval ? 1 + (A.num_betas - 1) / A.interval : 0;
    RingState rs;
    bool live = false;
    for (int64_t r = gw; r < A.num_samples; r += A.shared_stream ? 1 : warps) {
        if (!live) {  // cpu_rotormc.cpp:389-390
            ring_init(W.ring, rs, A.seeds[r], lane);
            live = A.shared_stream != 0;
        }
        uint8_t *row = A.rows + r * n;
        for (int v = (int)lane; v < n; v += 32) W.st[v] = row[v];
        __syncwarp();
        if (PROPOSAL <= 1) {
            for (int v = (int)lane; v < n; v += 32)
                W.de.set(v, __dmul_rn(rmc_field(W, v), __dmul_rn(-2.0, cs[W.st[v]])));
            __syncwarp();
        }
        ring_refill(W.ring, rs, lane);
        rs.q += 32;  // burn-in
        uint8_t *stats = A.stats ? A.stats + r * points * n : nullptr;
        for (int b = 0; b < A.num_betas; ++b) {
            const double beta = __ldg(&A.hp[b]);
            [[maybe_unused]] RmcProposal q;
            if constexpr (PROPOSAL >= 2) q = rmc_proposal<PROPOSAL>(beta, __ldg(&A.hd[b]));
            for (int sw = 0; sw < A.sweeps_per_beta; ++sw) {
                if constexpr (PROPOSAL <= 1) {
                    if constexpr (RANDOM_ORDER)
                        rmc_reflect_random<PROPOSAL == 0>(W, rs, beta, magic);
                    else
                        rmc_reflect_sequential<PROPOSAL == 0>(W, rs, beta);
                } else {
                    if constexpr (RANDOM_ORDER)
                        rmc_angle_random(W, rs, q, magic);
                    else
                        rmc_angle_sequential(W, rs, q);
                }
            }
            if (stats && b % A.interval == 0) {
                for (int v = (int)lane; v < n; v += 32) stats[v] = W.st[v];
                stats += n;
            }
        }
        __syncwarp();
        // cpu_rotormc.cpp:310-326: terms lane-parallel, the sum in order.
        double e = 0.0;
        for (int base = 0; base < n; base += 32) {
            const int v = base + (int)lane;
            const double t = v < n ? __dmul_rn(cs[W.st[v]], __ldg(&A.h[v])) : 0.0;
            const int cnt = min(32, n - base);
            for (int j = 0; j < cnt; ++j) e = __dadd_rn(e, __shfl_sync(kFull, t, j));
        }
        for (int64_t base = 0; base < A.m; base += 32) {
            const int64_t k = base + lane;
            double t = 0.0;
            if (k < A.m)
                t = __dmul_rn(__dmul_rn(cs[W.st[__ldg(&A.cu[k])]], __ldg(&A.cw[k])),
                              cs[W.st[__ldg(&A.cv[k])]]);
            const int cnt = (int)min((int64_t)32, A.m - base);
            for (int j = 0; j < cnt; ++j) e = __dadd_rn(e, __shfl_sync(kFull, t, j));
        }
        if (lane == 0) A.energies[r] = e;
        for (int v = (int)lane; v < n; v += 32) row[v] = W.st[v];
        __syncwarp();
    }
    if (W.near && lane == 0) atomicAdd(A.near, (unsigned long long)W.near);
}

// One thread per sample (see above).  Angles and delta energies are interleaved
// across samples (element (v, r) at v * num_samples + r), so in sequential order
// a warp's 32 samples touch one variable in one transaction.
template <bool RANDOM_ORDER, int PROPOSAL>
__global__ void __launch_bounds__(64) rmc_thread_kernel(RmcArgs A) {
    __shared__ double cs[256], sn[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        cs[i] = A.cos_table[i];
        sn[i] = A.sin_table[i];
    }
    __syncthreads();
    const int64_t R = A.num_samples;
    const int n = A.n;
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    const int points = A.interval ? 1 + (A.num_betas - 1) / A.interval : 0;
    const uint64_t magic = ~0ull / (uint64_t)n;
    unsigned near = 0;
    uint64_t s0 = A.seeds[r] ? A.seeds[r] : ~0ull, s1 = 0;  // cpu_rotormc.cpp:389-390
    uint8_t *st = A.states + r;  // element v at st[v * R]
    double *de = PROPOSAL <= 1 ? A.de + r : nullptr;
    uint8_t *row = A.rows + r * n;
    for (int v = 0; v < n; ++v) st[v * R] = row[v];
    auto field = [&](int var) {
        const uint2 vi = __ldg(&A.vinfo[var]);
        double e = __ldg(&A.h[var]);
        for (unsigned k = vi.x; k < vi.x + vi.y; ++k)
            e = __dadd_rn(e, __dmul_rn(cs[st[(int64_t)__ldg(&A.col[k]) * R]], __ldg(&A.w[k])));
        return e;
    };
    if constexpr (PROPOSAL <= 1) {
        for (int v = 0; v < n; ++v)
            de[v * R] = __dmul_rn(field(v), __dmul_rn(-2.0, cs[st[v * R]]));
    }
    for (int i = 0; i < 32; ++i) xs_advance(s0, s1);  // burn-in
    uint8_t *stats = A.stats ? A.stats + r * points * n : nullptr;
    for (int b = 0; b < A.num_betas; ++b) {
        const double beta = __ldg(&A.hp[b]);
        [[maybe_unused]] RmcProposal q;
        if constexpr (PROPOSAL >= 2) q = rmc_proposal<PROPOSAL>(beta, __ldg(&A.hd[b]));
        for (int sw = 0; sw < A.sweeps_per_beta; ++sw) {
            for (int i = 0; i < n; ++i) {
                const int var = RANDOM_ORDER ? mod_n(xs_next(s0, s1), (uint32_t)n, magic) : i;
                const uint8_t cur = st[var * R];
                if constexpr (PROPOSAL <= 1) {  // :167-196
                    const double d = de[var * R];
                    int x = 1;
                    if (PROPOSAL == 0)
                        x = rmc_gibbs(__dmul_rn(d, beta), xs_next(s0, s1));
                    else if (!(d <= 0.0))
                        x = rmc_metropolis(__dmul_rn(-d, beta), xs_next(s0, s1));
                    near += (unsigned)x >> 1;
                    if (!(x & 1)) continue;
                    const uint8_t prop = (uint8_t)(128 + cur);  // :270-283
                    const double mult = __dmul_rn(2.0, __dsub_rn(cs[cur], cs[prop]));
                    const uint2 vi = __ldg(&A.vinfo[var]);
                    for (unsigned k = vi.x; k < vi.x + vi.y; ++k) {
                        const int64_t nb = (int64_t)__ldg(&A.col[k]) * R;
                        de[nb] = __dadd_rn(
                            de[nb], __dmul_rn(__dmul_rn(mult, __ldg(&A.w[k])), cs[st[nb]]));
                    }
                    st[var * R] = prop;
                    de[var * R] = -d;
                } else {
                    const uint64_t r1 = xs_next(s0, s1);
                    const uint64_t r2 = q.tf ? xs_next(s0, s1) : 0;
                    const uint8_t prop = rmc_angle(q, cur, r1, r2);
                    const double dlm = rmc_log_ratio(q, field(var), __ldg(&A.tf[var]), cs[prop],
                                                     cs[cur], sn[prop], sn[cur]);
                    bool flip = dlm >= 0.0;
                    if (!flip) {
                        const int x = rmc_metropolis(dlm, xs_next(s0, s1));
                        flip = (x & 1) != 0;
                        near += (unsigned)x >> 1;
                    }
                    if (flip) st[var * R] = prop;
                }
            }
        }
        if (stats && b % A.interval == 0) {
            for (int v = 0; v < n; ++v) stats[v] = st[v * R];
            stats += n;
        }
    }
    double e = 0.0;  // cpu_rotormc.cpp:310-326
    for (int v = 0; v < n; ++v) e = __dadd_rn(e, __dmul_rn(cs[st[v * R]], __ldg(&A.h[v])));
    for (int64_t c = 0; c < A.m; ++c)
        e = __dadd_rn(e, __dmul_rn(__dmul_rn(cs[st[(int64_t)__ldg(&A.cu[c]) * R]], __ldg(&A.cw[c])),
                                   cs[st[(int64_t)__ldg(&A.cv[c]) * R]]));
    A.energies[r] = e;
    for (int v = 0; v < n; ++v) row[v] = st[v * R];
    if (near) atomicAdd(A.near, (unsigned long long)near);
}

}  // namespace b200sa
