// Path-integral Monte Carlo annealing (the reference's SQA localPIMC,
// dwave/samplers/sqa/src/localPIMC.cpp) on the GPU.  Included by
// sa_launch.cu next to the annealing kernels.
//
// An update draws a data-dependent number of random numbers (break proposals,
// one Gibbs draw per domain) from one mt19937 stream and merges variable-length
// break lists, so a sample is one sequential chain of updates, bound by the
// latency of one update; many samples run side by side.  Single-qubit updates
// run on a warp per sample (pimc_warp_kernel, below), chain updates, unusual
// inputs and calls of very many samples on one thread per sample.  Every sample
// keeps its world lines in global memory: the first Trotter slice (int8 spins), the
// number of breaks of each variable and their positions (cap_breaks slots per
// variable, increasing).  Every slot (thread) keeps its mt19937 state and a
// scratch area (proposals, interfaces, domain fields, chain labels).
//
// Arithmetic follows localPIMC.cpp operation for operation:
//   run (:126-157)              Hd sets Gamma, Hp sets invTemp per schedule step;
//                               sweeps_per_beta * n updates of uniformly drawn
//                               qubits (or chains) per step
//   qubitUpdate (:361-393), chainUpdate (:395-464), makeDomainGraph (:474-541)
//   addHToEffectiveField (:277-295), addJToEffectiveField (:297-359)
//   makeBreakProposals (:543-555), GibbsSamplePM1, pNotJoin (:568-576)
//   get_state_energy (:59-75)
// and std::mt19937 with libstdc++'s uniform_int_distribution (Lemire's
// method on the 64-bit product) and generate_canonical<double, 53>.
//
// Where the reference calls libm (log, tanh, exp) this calls CUDA's; every
// decision they feed is checked against a relative band of 2^-48 around its
// threshold and counted as a near tie (0 expected; the host reports them).
#pragma once
#include "sa_kernel.cuh"

namespace b200sa {

// mt19937 (Matsumoto & Nishimura 1998), regenerated one word per draw: word
// i is replaced by its successor from words i, i + 1 and i + 397 (mod 624) just
// before it is output.  Regenerating in index order is what the block
// regeneration of all 624 words does, so the stream is the same; the cost is
// the same for every draw, so threads of a warp never wait on one thread's
// 624-word burst.
struct PimcRng {
    uint32_t *mt;
    int idx;       // next word to regenerate and output
    uint32_t cur;  // mt[idx], not yet regenerated

    __device__ void seed(uint32_t s) {
        uint32_t x = s;
        mt[0] = x;
        for (int i = 1; i < kMtWords; ++i) {
            x = 1812433253u * (x ^ (x >> 30)) + (uint32_t)i;
            mt[i] = x;
        }
        idx = 0;
        cur = s;
    }
    __device__ __forceinline__ uint32_t next() {
        const int i1 = idx == kMtWords - 1 ? 0 : idx + 1;
        const int im = idx < kMtWords - 397 ? idx + 397 : idx - (kMtWords - 397);
        const uint32_t b = mt[i1];
        const uint32_t t = (cur & 0x80000000u) | (b & 0x7fffffffu);
        uint32_t y = mt[im] ^ (t >> 1) ^ ((t & 1u) ? 0x9908b0dfu : 0u);
        mt[idx] = y;
        idx = i1;
        cur = b;
        y ^= y >> 11;
        y ^= (y << 7) & 0x9d2c5680u;
        y ^= (y << 15) & 0xefc60000u;
        y ^= y >> 18;
        return y;
    }
    // generate_canonical<double, 53>: (d1 + d2 * 2^32) / 2^64, below 1.
    __device__ __forceinline__ double canonical() {
        const double lo = __uint2double_rn(next());
        const double hi = __uint2double_rn(next());
        const double r = __ddiv_rn(__dadd_rn(lo, __dmul_rn(hi, 4294967296.0)), kTwo64);
        return r >= 1.0 ? 0x1.fffffffffffffp-1 : r;  // nextafter(1, 0)
    }
    // uniform_int_distribution<int>(0, range - 1).
    __device__ __forceinline__ int below(uint32_t range) {
        uint64_t prod = (uint64_t)next() * range;
        uint32_t low = (uint32_t)prod;
        if (low < range) {
            const uint32_t threshold = (0u - range) % range;
            while (low < threshold) {
                prod = (uint64_t)next() * range;
                low = (uint32_t)prod;
            }
        }
        return (int)(prod >> 32);
    }
};

// The per-thread view of one sample's world lines.
struct PimcWorld {
    int8_t *s;        // [n]
    int32_t *cnt;     // [n]
    int32_t *brk;     // [n][stride], 16-byte aligned
    int cap, stride;
    double beta, gamma;
    unsigned near;
    bool overflow;

    __device__ const int32_t *list(int v) const { return brk + (int64_t)v * stride; }
    __device__ int32_t *list(int v) { return brk + (int64_t)v * stride; }
};

// makeBreakProposals: positions with exponential gaps of scale slices / Gamma.
__device__ int pimc_proposals(PimcRng &g, PimcWorld &W, int32_t *out, int cap) {
    const double neg_scale = -__ddiv_rn((double)kPimcSlices, W.gamma);
    int k = 0;
    double x = __dmul_rn(neg_scale, log(g.canonical()));
    double position = x;
    for (;;) {
        // int(position) and the bound both switch at integers.
        if (position < (double)(kPimcSlices + 1) && isfinite(position))
            W.near += fabs(position - rint(position)) <= fmax(fabs(x), 1.0) * kTieRel;
        if (!(position < (double)kPimcSlices)) break;
        if (k == cap) {
            W.overflow = true;
            return k;
        }
        out[k] = (int)position;
        x = __dmul_rn(neg_scale, log(g.canonical()));
        position = __dadd_rn(__dadd_rn(x, (double)out[k]), 1.0);
        ++k;
    }
    return k;
}

// std::merge(a, b): on equal values the element of a comes first.
__device__ int pimc_merge(const int32_t *a, int na, const int32_t *b, int nb, int32_t *out) {
    int i = 0, j = 0, k = 0;
    while (i < na && j < nb) out[k++] = b[j] < a[i] ? b[j++] : a[i++];
    while (i < na) out[k++] = a[i++];
    while (j < nb) out[k++] = b[j++];
    return k;
}

// Interfaces of qubit q: proposals merged with its breaks, or the single
// book-keeping value when there is at most one of them together.
__device__ int pimc_interfaces(PimcRng &g, PimcWorld &W, int q, int32_t *props, int cap_props,
                               int32_t *itf) {
    const int np = pimc_proposals(g, W, props, cap_props);
    const int nb = W.cnt[q];
    if (np + nb > 1) return pimc_merge(props, np, W.list(q), nb, itf);
    itf[0] = kPimcSlices;
    return 1;
}

// addHToEffectiveField; lab maps a domain to its accumulator (null: itself).
__device__ void pimc_add_h(double *eff, const int32_t *lab, const int32_t *itf, int nd,
                           double H) {
    H = __ddiv_rn(H, (double)kPimcSlices);
    const int d0 = lab ? lab[0] : 0;
    eff[d0] = __dadd_rn(eff[d0], __dmul_rn((double)(kPimcSlices + itf[0] - itf[nd - 1]), H));
    for (int i = 1; i < nd; ++i) {
        const int d = lab ? lab[i] : i;
        eff[d] = __dadd_rn(eff[d], __dmul_rn((double)(itf[i] - itf[i - 1]), H));
    }
}

// addJToEffectiveField: the neighbour's spin, flipped at each of its breaks,
// over the domains of this qubit.  The merged list (neighbour first on equal
// values) is walked without being stored.
__device__ void pimc_add_j(double *eff, const int32_t *lab, const int32_t *itf, int nd,
                           const int32_t *nbk, int nn, double Js) {
    Js = __ddiv_rn(Js, (double)kPimcSlices);
    int i = 0, j = 0;  // cursors into nbk and itf
    auto next = [&]() { return (i >= nn || (j < nd && itf[j] < nbk[i])) ? itf[j++] : nbk[i++]; };
    const int L = nn + nd;
    const int front = nn ? min(nbk[0], itf[0]) : itf[0];
    const int back = nn ? max(nbk[nn - 1], itf[nd - 1]) : itf[nd - 1];
    const int d0 = lab ? lab[0] : 0;
    eff[d0] = __dadd_rn(eff[d0], __dmul_rn((double)(kPimcSlices + front - back), Js));
    int cur = next();
    int k = 0, oi = 0;
    for (; k + 1 < L; ++k) {
        if (cur == itf[oi]) {
            if (++oi == nd) break;
        } else {
            Js = -Js;
        }
        const int nxt = next();
        const int d = lab ? lab[oi] : oi;
        eff[d] = __dadd_rn(eff[d], __dmul_rn((double)(nxt - cur), Js));
        cur = nxt;
    }
    for (; k + 1 < L; ++k) {
        const int nxt = next();
        eff[d0] = __dadd_rn(eff[d0], __dmul_rn((double)(nxt - cur), Js));
        Js = -Js;
        cur = nxt;
    }
}

// Adds h and every neighbour's world line of qubit q to the domain fields,
// neighbours in adjacency order.  The spin, break count and coupling of up
// to four neighbours are loaded before any field is written, so those loads
// overlap instead of waiting behind the previous neighbour's stores.
__device__ void pimc_fields(const PimcArgs &A, const PimcWorld &W, int q, double *eff,
                            const int32_t *lab, const int32_t *itf, int nd) {
    pimc_add_h(eff, lab, itf, nd, __ldg(&A.h[q]));
    const uint2 vi = __ldg(&A.vinfo[q]);
    const unsigned end = vi.x + vi.y;
    for (unsigned k0 = vi.x; k0 < end; k0 += 4) {
        int nb[4], cnt[4];
        double js[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) nb[j] = k0 + j < end ? __ldg(&A.col[k0 + j]) : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (k0 + j < end) {
                cnt[j] = W.cnt[nb[j]];
                js[j] = __dmul_rn((double)W.s[nb[j]], __ldg(&A.w[k0 + j]));
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (k0 + j < end) pimc_add_j(eff, lab, itf, nd, W.list(nb[j]), cnt[j], js[j]);
    }
}

__device__ __forceinline__ int pimc_gibbs(PimcRng &g, PimcWorld &W, double field) {
    const double thr = __dadd_rn(__dmul_rn(g.canonical(), 2.0), -1.0);  // uniform(-1, 1)
    const double t = tanh(__dmul_rn(W.beta, field));
    W.near += fabs(t - thr) <= fabs(t) * kTieRel;
    return t > thr ? -1 : 1;
}

// pNotJoin(overlaps) < uniform(0, 1)
__device__ __forceinline__ bool pimc_join(PimcRng &g, PimcWorld &W, double jchain, int overlaps) {
    const double p = exp(__ddiv_rn(
        __dmul_rn(__dmul_rn(__dmul_rn(2.0, jchain), (double)overlaps), W.beta),
        (double)kPimcSlices));
    const double c = g.canonical();
    W.near += fabs(p - c) <= p * kTieRel;
    return p < c;
}

// Rewrites the breaks of qubit q from its interfaces and the spins of its
// domains; returns false (overflow) when they do not fit.
template <typename SPIN>
__device__ bool pimc_store(PimcWorld &W, int q, const int32_t *itf, int nd, SPIN spin) {
    const int first = spin(0);
    W.s[q] = (int8_t)first;
    int32_t *out = W.list(q);
    int c = 0, sv = first;
    for (int d = 1; d < nd; ++d) {
        if (sv * spin(d) != 1) {
            sv = -sv;
            if (c == W.cap) return false;
            out[c++] = itf[d - 1];
        }
    }
    if (sv != first) {
        if (c == W.cap) return false;
        out[c++] = itf[nd - 1];
    }
    W.cnt[q] = c;
    return true;
}

// qubitUpdate (localPIMC.cpp:361-393).  Gibbs draws go domain by domain in
// order, so drawing them all before rewriting the breaks keeps the stream.
__device__ void pimc_qubit_update(const PimcArgs &A, PimcRng &g, PimcWorld &W, int sp,
                                  int32_t *props, int32_t *itf, int32_t *sv, double *eff) {
    const int nd = pimc_interfaces(g, W, sp, props, A.cap_props, itf);
    if (W.overflow) return;
    for (int i = 0; i < nd; ++i) eff[i] = 0.0;
    pimc_fields(A, W, sp, eff, nullptr, itf, nd);
    for (int d = 0; d < nd; ++d) sv[d] = pimc_gibbs(g, W, eff[d]);
    if (!pimc_store(W, sp, itf, nd, [&](int d) { return sv[d]; })) W.overflow = true;
}

__device__ __forceinline__ int pimc_find(int32_t *parent, int x) {
    while (parent[x] != x) {
        parent[x] = parent[parent[x]];
        x = parent[x];
    }
    return x;
}

// Parents always point to smaller indices, so pimc_find ends.
__device__ __forceinline__ void pimc_union(int32_t *parent, int a, int b) {
    a = pimc_find(parent, a);
    b = pimc_find(parent, b);
    if (a != b) parent[max(a, b)] = min(a, b);
}

// makeDomainGraph (localPIMC.cpp:474-541) for chain qubits c and c + 1:
// joins go straight into a union-find forest over the domains.
__device__ void pimc_domain_graph(const PimcArgs &A, PimcRng &g, PimcWorld &W, int sp, int c,
                                  const int32_t *itfA, int nA, int z, const int32_t *itfB,
                                  int nB, int f, int32_t *pair, int32_t *parent) {
    const int q = sp * A.qpc + c;
    int s0s1 = (int)W.s[q] * (int)W.s[q + 1];
    int L = pimc_merge(itfA, nA, itfB, nB, pair);
    if (pair[0] == kPimcSlices) {
        if (s0s1 == 1 && pimc_join(g, W, A.jchain, kPimcSlices)) pimc_union(parent, z, f);
        return;
    }
    if (pair[L - 1] == kPimcSlices) --L;
    if (s0s1 == 1 && pimc_join(g, W, A.jchain, kPimcSlices - pair[L - 1] + pair[0]))
        pimc_union(parent, z, f);
    const int32_t *b0 = W.list(q), *b1 = W.list(q + 1);
    const int n0 = W.cnt[q], n1 = W.cnt[q + 1];
    int p0 = 0, e0 = 0, p1 = 0, e1 = 0;
    bool valid0 = itfA[0] != kPimcSlices;
    for (int i = 1; i < L; ++i) {
        if (valid0 && pair[i - 1] == itfA[p0]) {
            if (nA == ++p0) {
                valid0 = false;
                p0 = 0;
            }
            if (n0 > e0 && pair[i - 1] == b0[e0]) {
                s0s1 = -s0s1;
                ++e0;
            }
        } else {
            if (nB == ++p1) p1 = 0;
            if (n1 > e1 && pair[i - 1] == b1[e1]) {
                s0s1 = -s0s1;
                ++e1;
            }
        }
        if (s0s1 == 1 && pimc_join(g, W, A.jchain, pair[i] - pair[i - 1]))
            pimc_union(parent, z + p0, f + p1);
    }
}

// chainUpdate (localPIMC.cpp:395-464).  Components are numbered in order of
// their smallest domain, as the reference's depth-first labelling from roots
// 0, 1, ... numbers them.  Scratch: itf [Q][C], off [Q + 1], lab / parent /
// sv [Q * C], pair [2C], eff [Q * C].
__device__ void pimc_chain_update(const PimcArgs &A, PimcRng &g, PimcWorld &W, int sp,
                                  int32_t *props, int32_t *itf, int32_t *off, int32_t *lab,
                                  int32_t *parent, int32_t *sv, int32_t *pair, double *eff) {
    const int Q = A.qpc;
    const int C = A.cap_props + A.cap_breaks;
    int total = 0;
    for (int c = 0; c < Q; ++c) {
        const int nd = pimc_interfaces(g, W, Q * sp + c, props, A.cap_props, itf + c * C);
        if (W.overflow) return;
        off[c] = total;
        total += nd;
    }
    off[Q] = total;
    for (int d = 0; d < total; ++d) parent[d] = d;
    for (int c = 0; c + 1 < Q; ++c)
        pimc_domain_graph(A, g, W, sp, c, itf + c * C, off[c + 1] - off[c], off[c],
                          itf + (c + 1) * C, off[c + 2] - off[c + 1], off[c + 1], pair, parent);
    int ncomp = 0;
    for (int d = 0; d < total; ++d) sv[d] = -1;  // label of each root
    for (int d = 0; d < total; ++d) {
        const int r = pimc_find(parent, d);
        if (sv[r] < 0) sv[r] = ncomp++;
        lab[d] = sv[r];
    }
    for (int k = 0; k < ncomp; ++k) eff[k] = 0.0;
    for (int c = 0; c < Q; ++c) {
        pimc_fields(A, W, Q * sp + c, eff, lab + off[c], itf + c * C, off[c + 1] - off[c]);
    }
    for (int k = 0; k < ncomp; ++k) sv[k] = pimc_gibbs(g, W, eff[k]);
    for (int c = 0; c < Q; ++c) {
        const int *l = lab + off[c];
        if (!pimc_store(W, Q * sp + c, itf + c * C, off[c + 1] - off[c],
                        [&](int d) { return sv[l[d]]; })) {
            W.overflow = true;
            return;
        }
    }
}

template <bool CHAIN>
__global__ void __launch_bounds__(64) pimc_kernel(PimcArgs A) {
    const int R = A.num_samples;
    const int n = A.n;
    const int slot = A.shared_stream ? 0 : (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (slot >= R) return;
    if (A.shared_stream && (blockIdx.x != 0 || threadIdx.x != 0)) return;
    const int first = slot;
    const int last = A.shared_stream ? R : first + 1;
    const int points = A.interval ? 1 + (A.num_betas - 1) / A.interval : 0;
    const int Q = CHAIN ? A.qpc : 1;
    const int C = A.cap_props + A.cap_breaks;
    int32_t *si = A.scratch_i + (int64_t)slot * A.scratch_ints;
    int32_t *props = si;
    int32_t *itf = props + A.cap_props;
    int32_t *sv = itf + Q * C;
    int32_t *off = sv + Q * C;
    int32_t *lab = off + Q + 1;
    int32_t *parent = lab + Q * C;
    int32_t *pair = parent + Q * C;
    double *eff = A.scratch_d + (int64_t)slot * A.scratch_doubles;
    PimcRng g;
    g.mt = A.mt + (int64_t)slot * kMtWords;
    PimcWorld W;
    W.cap = A.cap_breaks;
    W.stride = A.list_stride;
    W.near = 0;
    W.overflow = false;
    for (int r = first; r < last && !W.overflow; ++r) {
        if (r == first) g.seed(A.seeds[A.shared_stream ? 0 : r]);  // localPIMC.cpp:578-587
        W.s = A.states + (int64_t)r * n;
        W.cnt = A.counts + (int64_t)r * n;
        W.brk = A.breaks + (int64_t)r * n * A.list_stride;
        int8_t *stats = A.stats ? A.stats + (int64_t)r * points * n : nullptr;
        for (int b = 0; b < A.num_betas && !W.overflow; ++b) {
            W.gamma = __ldg(&A.hd[b]);
            W.beta = __ldg(&A.hp[b]);
            const int64_t updates = (int64_t)A.sweeps_per_beta * n;
            for (int64_t k = 0; k < updates && !W.overflow; ++k) {
                if (CHAIN)
                    pimc_chain_update(A, g, W, g.below((uint32_t)A.chains), props, itf, off, lab,
                                      parent, sv, pair, eff);
                else
                    pimc_qubit_update(A, g, W, g.below((uint32_t)n), props, itf, sv, eff);
            }
            if (stats && b % A.interval == 0) {
                for (int v = 0; v < n; ++v) stats[v] = W.s[v];
                stats += n;
            }
        }
        double e = 0.0;  // localPIMC.cpp:59-75
        for (int v = 0; v < n; ++v)
            e = __dadd_rn(e, __dmul_rn((double)W.s[v], __ldg(&A.h[v])));
        for (int64_t c = 0; c < A.m; ++c)
            e = __dadd_rn(e, __dmul_rn(__dmul_rn((double)W.s[__ldg(&A.cu[c])], __ldg(&A.cw[c])),
                                       (double)W.s[__ldg(&A.cv[c])]));
        A.energies[r] = e;
    }
    if (W.overflow) atomicExch(A.overflow, 1);
    if (W.near) atomicAdd(A.near, (unsigned long long)W.near);
}

// ---- Single-qubit updates by a warp per sample --------------------------------
// The lanes of a warp generate the mt19937 words side by side (the state in
// shared memory), take the logarithms of 32 proposals at once, merge by rank,
// and own one domain each, whose field they add up over the neighbours' breaks
// and whose spin they draw.  An update takes about 900 warp instructions, which
// is what bounds it: 6 cycles each for few samples (with one thread per sample
// the latency of dependent loads, about 50,000 cycles an update), the issue
// slots (70% busy) from about 4000 samples on.  Measured, n = 512 6-regular, field
// 5 -> 0.05, 16 steps: 4096 samples 209 ms with one thread per sample, 118 ms with
// four samples to a warp (8 lanes each; the samples of a warp diverge), 40 ms with
// a warp; 8 steps: 1000 samples 107 -> 15 ms, 16384 139 -> 78 ms.  From
// pimc_thread_samples on the thread per sample is the faster one.

// mt19937 as a ring in shared memory: slot k mod 624 is replaced in place by
// word k + 624, 32 words at a time and only a few ahead of the draws.
struct PimcWarpRng {
    uint32_t *mt;
    int pos;    // slot of the next word to draw
    int avail;  // words generated from there on
    int lane;

    static __device__ __forceinline__ int wrap(int i) {
        return i >= kMtWords ? i - kMtWords : i;
    }
    __device__ void seed(uint32_t s) {
        __syncwarp();
        uint32_t x = s;
        if (lane == 0) mt[0] = x;
        for (int i = 1; i < kMtWords; ++i) {
            x = 1812433253u * (x ^ (x >> 30)) + (uint32_t)i;
            if (lane == (i & 31)) mt[i] = x;
        }
        pos = 0;
        avail = 0;
        __syncwarp();
    }
    // At least k words ahead (k <= kMtWords - 32).
    __device__ __forceinline__ void ensure(int k) {
        while (avail < k) {
            const int i = wrap(wrap(pos + avail) + lane);
            const uint32_t t = (mt[i] & 0x80000000u) | (mt[wrap(i + 1)] & 0x7fffffffu);
            const uint32_t y =
                mt[wrap(i + 397)] ^ (t >> 1) ^ ((t & 1u) ? 0x9908b0dfu : 0u);
            __syncwarp();
            mt[i] = y;
            avail += 32;
            __syncwarp();
        }
    }
    __device__ __forceinline__ void consume(int k) {
        pos = wrap(pos + k);
        avail -= k;
    }
    // The word o draws ahead.
    __device__ __forceinline__ uint32_t word(int o) const {
        uint32_t y = mt[wrap(pos + o)];
        y ^= y >> 11;
        y ^= (y << 7) & 0x9d2c5680u;
        y ^= (y << 15) & 0xefc60000u;
        y ^= y >> 18;
        return y;
    }
    // See PimcRng::canonical; the division by 2^64 is exact as a product.
    __device__ __forceinline__ double canonical(int o) const {
        const double lo = __uint2double_rn(word(o));
        const double hi = __uint2double_rn(word(o + 1));
        const double r = __dmul_rn(__dadd_rn(lo, __dmul_rn(hi, 4294967296.0)), 0x1p-64);
        return r >= 1.0 ? 0x1.fffffffffffffp-1 : r;
    }
    __device__ __forceinline__ int below(uint32_t range) {
        ensure(1);
        uint64_t prod = (uint64_t)word(0) * range;
        consume(1);
        if ((uint32_t)prod < range) {
            const uint32_t threshold = (0u - range) % range;
            while ((uint32_t)prod < threshold) {
                ensure(1);
                prod = (uint64_t)word(0) * range;
                consume(1);
            }
        }
        return (int)(prod >> 32);
    }
};

// A warp's scratch: 32 neighbours (s J / 65536, variable, number of
// breaks), proposals, the qubit's breaks, interfaces, spins.
struct PimcWarpScratch {
    double *js;
    int32_t *nx, *nn;
    int32_t *props, *own, *itf;
    int8_t *sv;
};

// The gaps between break proposals at transverse field gamma: -scale, and a
// bound below which a first uniform number c leaves no proposal for certain
// (-65536 / gamma log(c) is beyond 65537, so its tie band holds no slice
// either), without taking its logarithm.
struct PimcGap {
    double neg_scale, none;
};
__device__ __forceinline__ PimcGap pimc_gap(double gamma) {
    PimcGap p;
    p.neg_scale = -__ddiv_rn((double)kPimcSlices, gamma);
    p.none = gamma >= 0.0 && gamma < 700.0
                 ? exp(-gamma * (1.0 + 1.0 / kPimcSlices)) * (1.0 - 1e-9)
                 : -1.0;
    return p;
}

// makeBreakProposals: the next 32 gaps are drawn side by side, their
// positions follow one after another.  Returns -1 when they do not fit.
__device__ __forceinline__ int pimc_warp_proposals(PimcWarpRng &g, unsigned &near,
                                                    const PimcGap &gap, int32_t *props, int cap) {
    g.ensure(2);
    if (g.canonical(0) < gap.none) {
        g.consume(2);
        return 0;
    }
    int k = 0, last = 0;
    for (;;) {
        g.ensure(64);
        const double mine = __dmul_rn(gap.neg_scale, log(g.canonical(2 * g.lane)));
        for (int j = 0; j < 32; ++j) {
            const double x = __shfl_sync(kFull, mine, j);
            const double position =
                k == 0 ? x : __dadd_rn(__dadd_rn(x, (double)last), 1.0);
            // (The tie band of a position is below 1e-9, see pimc_proposals.)
            const int slice = (int)position;
            const double part = position - (double)slice;
            if (!(part > 1e-9 && part < 1.0 - 1e-9) &&
                position < (double)(kPimcSlices + 1) && isfinite(position))
                near += g.lane == 0 &&
                        fabs(position - rint(position)) <= fmax(fabs(x), 1.0) * kTieRel;
            if (!(position < (double)kPimcSlices)) {
                g.consume(2 * (j + 1));
                return k;
            }
            if (k == cap) return -1;
            last = slice;
            if (g.lane == 0) props[k] = last;
            ++k;
        }
        g.consume(64);
    }
}

// One neighbour's world line (its nn > 0 breaks, in order) over the domain
// (lo, hi] of this lane.  pimc_add_j's additions to one domain are these, in
// this order; terms of length zero, where a break meets an interface, change
// nothing and are left out.  Domain `first` wraps around: the part from the
// last break or interface to the first one, the rest up to its interface
// (hi, with lo = -1), and the breaks beyond the last interface `tail`.  The
// sign before break j is that of j flips.
__device__ __forceinline__ double pimc_warp_add_j(double eff, bool first, int lo, int hi,
                                                   int tail, const int32_t *brk, int nn,
                                                   double Js) {
    const int bound = first ? tail : lo;
    int c = 0;
    for (int j = 0; j < nn; ++j) c += brk[j] <= bound;
    if (first) {
        const int front = min(brk[0], hi), back = max(brk[nn - 1], tail);
        eff = __dadd_rn(eff, __dmul_rn((double)(kPimcSlices + front - back), Js));
    }
    const double behind = (c & 1) ? -Js : Js;  // sign after `bound`
    double s = first ? Js : behind;
    bool open = !first;
    int cur = lo;
    for (int j = first ? 0 : c; j < nn; ++j) {
        const int x = brk[j];
        if (x >= hi) break;
        if (open) eff = __dadd_rn(eff, __dmul_rn((double)(x - cur), s));
        open = true;
        cur = x;
        s = -s;
    }
    if (open) eff = __dadd_rn(eff, __dmul_rn((double)(hi - cur), s));
    if (first) {
        s = behind;
        cur = tail;
        for (int j = c; j < nn; ++j) {
            const int x = brk[j];
            eff = __dadd_rn(eff, __dmul_rn((double)(x - cur), s));
            cur = x;
            s = -s;
        }
    }
    return eff;
}

// The same for one to four breaks b (unused ones beyond every slice): the
// sign before break j is fixed by j, so there is nothing to count or to loop
// over.
__device__ __forceinline__ double pimc_warp_add_j4(double eff, bool first, int lo, int hi,
                                                   int tail, int4 b, int back, double Js) {
    if (first)
        eff = __dadd_rn(eff, __dmul_rn((double)(kPimcSlices + min(b.x, hi) - max(back, tail)), Js));
    const int x[4] = {b.x, b.y, b.z, b.w};
    bool open = !first;
    int cur = lo;
    double s = Js;  // sign after the breaks below hi
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= 2 && x[j] > back) break;
        if (x[j] < hi) {
            s = j & 1 ? Js : -Js;
            if (x[j] > lo) {
                if (open)
                    eff = __dadd_rn(eff, __dmul_rn((double)(x[j] - cur), j & 1 ? -Js : Js));
                open = true;
                cur = x[j];
            }
        }
    }
    if (open) eff = __dadd_rn(eff, __dmul_rn((double)(hi - cur), s));
    if (back > tail && first) {
        cur = tail;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (x[j] > cur && x[j] <= back) {
                eff = __dadd_rn(eff, __dmul_rn((double)(x[j] - cur), j & 1 ? -Js : Js));
                cur = x[j];
            }
        }
    }
    return eff;
}

// pimc_gibbs on the uniform number c: tanh(x) > 2c - 1 is 2x log2(e) >
// log2(c / (1 - c)), which single precision decides outside a band of 2^-10
// (errors below 2^-14 for |x| < 12, where both sides are below 35); tanh and
// the draw then differ by more than 5e-14, far above tanh's error and the tie
// band.  From |x| = 12 on tanh is within 1e-10 of +-1.  Inside the band the
// exact comparison decides.  The new spin, or 0 inside the band.
__device__ __forceinline__ int pimc_gibbs_fast(double x, double c) {
    if (fabs(x) < 12.0) {
        const float l = __fmul_rn(2.0f * kLog2e, (float)x);
        const float y = lg2_approx((float)c) - lg2_approx((float)(1.0 - c));
        if (l > y + kBand) return -1;
        if (l < y - kBand) return 1;
    } else if (c > 1e-9 && c < 1.0 - 1e-9 && fabs(x) < 1e300) {
        return x > 0.0 ? -1 : 1;
    }
    return 0;
}

// The new spin, near ties in `near`.
__device__ __forceinline__ int pimc_gibbs_draw(double x, double c, unsigned &near) {
    const int fast = pimc_gibbs_fast(x, c);
    if (fast) return fast;
    const double thr = __dadd_rn(__dmul_rn(c, 2.0), -1.0);  // uniform(-1, 1)
    const double t = tanh(x);
    near += fabs(t - thr) <= fabs(t) * kTieRel;
    return t > thr ? -1 : 1;
}

// qubitUpdate (localPIMC.cpp:361-393) of qubit q; false when a capacity would
// be exceeded.
__device__ __forceinline__ bool pimc_warp_update(const PimcArgs &A, PimcWarpRng &g,
                                                  PimcWorld &W, const PimcWarpScratch &S,
                                                  const PimcGap &gap, int q) {
    const int lane = g.lane;
    const uint2 vi = __ldg(&A.vinfo[q]);
    const unsigned end = vi.x + vi.y;
    const double h = __ldg(&A.h[q]);
    const int nb = W.cnt[q];
    int32_t *brk = W.list(q);
    // Neighbours, one per lane: bit k of the result is set when neighbour
    // k0 + k has breaks.
    auto neighbours = [&](unsigned k0) {
        int cnt = 0;
        if (k0 + lane < end) {
            const int x = __ldg(&A.col[k0 + lane]);
            cnt = W.cnt[x];
            if (cnt) prefetch_l1(W.list(x));
            S.nx[lane] = x;
            S.nn[lane] = cnt;
            S.js[lane] = __dmul_rn(__dmul_rn((double)W.s[x], __ldg(&A.w[k0 + lane])),
                                 1.0 / kPimcSlices);
        }
        return __ballot_sync(kFull, cnt > 0);
    };
    unsigned broken = neighbours(vi.x);
    for (int j = lane; j < nb; j += 32) S.own[j] = brk[j];
    const int np = pimc_warp_proposals(g, W.near, gap, S.props, A.cap_props);
    if (np < 0) return false;
    __syncwarp();
    // Interfaces (pimc_interfaces): on equal values a proposal goes first.
    int nd = np + nb;
    const int32_t *itf = nb ? S.own : S.props;
    if (nd <= 1) {
        nd = 1;
        if (lane == 0) S.itf[0] = kPimcSlices;
        itf = S.itf;
    } else if (np && nb) {
        for (int k = lane; k < np; k += 32) {
            const int p = S.props[k];
            int c = k;
            for (int j = 0; j < nb; ++j) c += S.own[j] < p;
            S.itf[c] = p;
        }
        for (int j = lane; j < nb; j += 32) {
            const int b = S.own[j];
            int c = j;
            for (int k = 0; k < np; ++k) c += S.props[k] <= b;
            S.itf[c] = b;
        }
        itf = S.itf;
    }
    __syncwarp();
    // Fields and Gibbs draws, one domain per lane.
    const int tail = itf[nd - 1];
    for (int base = 0; base < nd; base += 32) {
        const int d = base + lane;
        const bool first = d == 0;
        const int lo = d > 0 && d <= nd ? itf[d - 1] : -1;
        const int hi = d < nd ? itf[d] : lo;
        const double len = (double)(first ? kPimcSlices + hi - tail : hi - lo);
        double eff = __dadd_rn(0.0, __dmul_rn(len, __dmul_rn(h, 1.0 / kPimcSlices)));
        for (unsigned k0 = vi.x; k0 < end; k0 += 32) {
            if (vi.y > 32u && (k0 != vi.x || base > 0)) {
                __syncwarp();
                broken = neighbours(k0);
                __syncwarp();
            }
            const int m = (int)min(32u, end - k0);
            for (int k = 0; k < m; ++k) {
                const double J = S.js[k];
                if (!((broken >> k) & 1u)) {
                    eff = __dadd_rn(eff, __dmul_rn(len, J));
                    continue;
                }
                const int32_t *list = W.list(S.nx[k]);
                const int nn = S.nn[k];
                if (nn <= 4) {
                    int4 x = *reinterpret_cast<const int4 *>(list);
                    const int back = nn == 1 ? x.x : nn == 2 ? x.y : nn == 3 ? x.z : x.w;
                    if (nn < 2) x.y = 2 * kPimcSlices;
                    if (nn < 3) x.z = 2 * kPimcSlices;
                    if (nn < 4) x.w = 2 * kPimcSlices;
                    eff = pimc_warp_add_j4(eff, first, lo, hi, tail, x, back, J);
                } else {
                    eff = pimc_warp_add_j(eff, first, lo, hi, tail, list, nn, J);
                }
            }
        }
        const int here = min(32, nd - base);
        g.ensure(2 * here);
        if (d < nd) {
            S.sv[d] = (int8_t)pimc_gibbs_draw(__dmul_rn(W.beta, eff), g.canonical(2 * lane), W.near);
        }
        g.consume(2 * here);
        __syncwarp();
    }
    // pimc_store: a break at the end of every domain whose successor differs.
    int c = 0;
    for (int base = 0; nd > 1 && base < nd; base += 32) {
        const int d = base + lane;
        const bool is =
            d < nd && S.sv[d] != S.sv[d + 1 < nd ? d + 1 : 0];
        const unsigned m = __ballot_sync(kFull, is);
        if (c + __popc(m) > W.cap) return false;
        if (is) brk[c + __popc(m & ((1u << lane) - 1u))] = itf[d];
        c += __popc(m);
    }
    if (lane == 0) {
        W.s[q] = S.sv[0];
        W.cnt[q] = c;
    }
    __syncwarp();
    return true;
}

// 64 registers: 32 warps per SM.
__global__ void __launch_bounds__(32 * kPimcMaxWarps, 8)
    pimc_warp_kernel(PimcArgs A, int warp_bytes) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int wid = (int)(threadIdx.x >> 5);
    const int64_t slot = (int64_t)blockIdx.x * (blockDim.x >> 5) + wid;
    const int R = A.num_samples, n = A.n;
    if (slot >= (A.shared_stream ? 1 : R)) return;
    const int last = A.shared_stream ? R : (int)slot + 1;
    const int points = A.interval ? 1 + (A.num_betas - 1) / A.interval : 0;
    PimcWarpRng g;
    g.lane = (int)(threadIdx.x & 31u);
    uint8_t *mem = smem + (size_t)wid * (size_t)warp_bytes;
    g.mt = reinterpret_cast<uint32_t *>(mem);
    PimcWarpScratch S;
    S.js = reinterpret_cast<double *>(g.mt + kMtWords);
    S.nx = reinterpret_cast<int32_t *>(S.js + 32);
    S.nn = S.nx + 32;
    S.props = S.nn + 32;
    S.own = S.props + A.cap_props;
    S.itf = S.own + A.cap_breaks;
    S.sv = reinterpret_cast<int8_t *>(S.itf + A.cap_props + A.cap_breaks);
    PimcWorld W;
    W.cap = A.cap_breaks;
    W.stride = A.list_stride;
    W.near = 0;
    W.overflow = false;
    for (int r = (int)slot; r < last && !W.overflow; ++r) {
        if (r == slot) g.seed(A.seeds[A.shared_stream ? 0 : r]);  // localPIMC.cpp:578-587
        W.s = A.states + (int64_t)r * n;
        W.cnt = A.counts + (int64_t)r * n;
        W.brk = A.breaks + (int64_t)r * n * A.list_stride;
        int8_t *stats = A.stats ? A.stats + (int64_t)r * points * n : nullptr;
        for (int b = 0; b < A.num_betas && !W.overflow; ++b) {
            const PimcGap gap = pimc_gap(__ldg(&A.hd[b]));
            W.beta = __ldg(&A.hp[b]);
            const int64_t updates = (int64_t)A.sweeps_per_beta * n;
            for (int64_t k = 0; k < updates && !W.overflow; ++k)
                W.overflow = !pimc_warp_update(A, g, W, S, gap, g.below((uint32_t)n));
            if (stats && b % A.interval == 0) {
                for (int v = g.lane; v < n; v += 32) stats[v] = W.s[v];
                stats += n;
            }
        }
        // localPIMC.cpp:59-75: terms side by side, the sum in order.
        double e = 0.0;
        for (int64_t base = 0; base < (int64_t)n + A.m; base += 32) {
            const int64_t i = base + g.lane, c = i - n;
            double t = 0.0;
            if (i < n)
                t = __dmul_rn((double)W.s[i], __ldg(&A.h[i]));
            else if (c < A.m)
                t = __dmul_rn(__dmul_rn((double)W.s[__ldg(&A.cu[c])], __ldg(&A.cw[c])),
                              (double)W.s[__ldg(&A.cv[c])]);
            const int cnt = (int)min((int64_t)32, (int64_t)n + A.m - base);
            for (int j = 0; j < cnt; ++j) e = __dadd_rn(e, __shfl_sync(kFull, t, j));
        }
        if (g.lane == 0) A.energies[r] = e;
    }
    if (W.overflow && g.lane == 0) atomicExch(A.overflow, 1);
    if (W.near) atomicAdd(A.near, (unsigned long long)W.near);
}

}  // namespace b200sa
