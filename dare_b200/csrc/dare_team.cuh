// dare_team.cuh -- a BiCGStab(2) solve that runs to its end inside one kernel.
//
// A team of thread blocks owns a system: every block a contiguous range of
// its cells.  The five kernels of an iteration (dare_march.cuh) become five
// passes over the block's cells, and the launch between two of them becomes
// one exchange in the team: it sums the pass's dot products and makes every
// block's stores visible to the others.  Two kinds of team:
//   * GridTeam: the blocks of a cooperative launch (all of them resident);
//   * ClusterTeam: the blocks of a thread-block cluster (hardware barrier,
//     partial sums through distributed shared memory).
// The sums are taken in block order, so results do not depend on timing, and
// every block evaluates the scalar recurrence itself on its own copy of the
// state, from the same totals.
//
// What it is for: systems whose passes are shorter than a kernel launch.  The
// vectors then stay in L2, so a pass costs its instructions and one exchange
// instead of a launch, a queue of work items and a DRAM pipeline.
#pragma once

#include "dare_march.cuh"

namespace dare_gpu {

constexpr int kTeamMaxBlocks = 160;   // blocks of a grid team
constexpr int kClusterMaxBlocks = 16; // blocks of a cluster team (the largest cluster)
constexpr int kTeamPolls = 1 << 22;   // polls of a wait before the block gives up, unless the context has a limit of its own

__device__ __forceinline__ double team_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }

// Sums of Q values over a warp, red[q * 32 + warp] written by one lane each.
// Several values share the shuffles: at each step a lane hands over the half
// of its values that the other lane will sum (5 values: 8 shuffles, not 25;
// a double costs two of the SM's 32 lanes a clock, and 32 warps wait for it).
template <int Q>
__device__ __forceinline__ void team_warp_sums(const double (&v)[Q], double* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if constexpr (Q == 1) {
        double a = v[0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += team_xor(a, o);
        if (lane == 0) red[wid] = a;
    } else if constexpr (Q == 2) {
        const bool h = lane & 16;
        double a = h ? v[1] : v[0];
        a += team_xor(h ? v[0] : v[1], 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) a += team_xor(a, o);
        if ((lane & 15) == 0) red[(h ? 32 : 0) + wid] = a;
    } else {
        static_assert(Q == 5, "one, two or five values");
        // lanes 0-15 keep values 0, 1, 2 and lanes 16-31 values 3, 4; then by
        // bit 3 the pair (0, 1) or 2, the pair (3, 4) or none; then by bit 2
        const bool h = lane & 16, h8 = lane & 8, h4 = lane & 4;
        double k0 = h ? v[3] : v[0], k1 = h ? v[4] : v[1], k2 = h ? 0. : v[2];
        k0 += team_xor(h ? v[0] : v[3], 16);
        k1 += team_xor(h ? v[1] : v[4], 16);
        k2 += team_xor(h ? v[2] : 0., 16);
        double m0 = h8 ? k2 : k0, m1 = h8 ? 0. : k1;
        m0 += team_xor(h8 ? k0 : k2, 8);
        m1 += team_xor(h8 ? k1 : 0., 8);
        double a = h4 ? m1 : m0;
        a += team_xor(h4 ? m0 : m1, 4);
        a += team_xor(a, 2);
        a += team_xor(a, 1);
        const int q = (h ? 3 : 0) + (h8 ? 2 : 0) + (h4 ? 1 : 0);
        if ((lane & 3) == 0 && !(h8 && (h4 || h))) red[q * 32 + wid] = a;
    }
}

// Block part of a sum: afterwards warp q (q < Q) holds the block's sum of
// value q in every lane.  The barrier inside also orders every store of the
// block before what those warps do next.
template <int Q>
__device__ __forceinline__ double team_block_sum(const double (&v)[Q], double* red /* [32 * kMaxQ] */) {
    team_warp_sums<Q>(v, red);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double a = 0.;
    if (wid < Q) {
        a = lane < ((int)blockDim.x >> 5) ? red[wid * 32 + lane] : 0.;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += team_xor(a, o);
    }
    return a;
}

// A grid team's buffer in global memory: per value a counter of arrivals on a
// line of its own, the arrivals at the end of the last launch, and two sets
// (a block can be one exchange ahead of another at most, which still reads
// the other set) of partial sums and of totals.  A total is stored as its two
// halves, each beside the low word of the counter's value it belongs to:
// 8-byte accesses are single, so a reader that finds that word in both has it.
struct TeamBuffer {
    struct {
        unsigned n, pad[31];
    } arrived[kMaxQ];
    unsigned base[kMaxQ], set;
    struct {
        unsigned long long half[2], pad[14];
    } total[2][kMaxQ];
    double parts[2][kMaxQ][kTeamMaxBlocks];
};

// Shared-memory scratch of a team's exchanges.
struct TeamShared {
    double red[32 * kMaxQ];
    double tot[kMaxQ];
    unsigned target[kMaxQ];
    int timeout, limit;
    double parts[2][kMaxQ][kClusterMaxBlocks];   // cluster teams: the blocks' sums, stored here by each of them
};

// The blocks of a cooperative launch.  Value q is handled by warp q of every
// block: it stores the block's sum and counts itself in; the last one adds the
// sums in block order and publishes the total the others wait for.  148
// blocks that all read all 148 partial sums queue at the few L2 slices that
// hold them (4000 cycles on top of 1200, every other exchange), which is why
// one does.
// Every wait ends: after `limit` polls the block gives up, and so do the
// blocks that wait for it.  (limit 0, a test's: it gives up at its first
// exchange, after counting itself in.)  The limit is read from shared memory:
// kept in a register of the loop it made the 64^3 solve 143 us for 140.
struct GridTeam {
    TeamBuffer* buf;
    TeamShared* sh;
    int rank, size, limit;
    unsigned set;   // partial-sum set of the last exchange

    __device__ void start() {   // before the block's first barrier
        if (threadIdx.x < kMaxQ) sh->target[threadIdx.x] = buf->base[threadIdx.x];
        if (threadIdx.x == 0) {
            sh->timeout = limit == 0;
            sh->limit = limit;
        }
        set = buf->set;
    }
    __device__ void stop() {    // after the last exchange
        if (rank == 0 && threadIdx.x < kMaxQ) buf->base[threadIdx.x] = sh->target[threadIdx.x];
        if (rank == 0 && threadIdx.x == 0) buf->set = set;
    }
    // The totals of Q values to fin(tot) in thread 0, then a barrier of the
    // block: what any block stored before its call is visible to all.  False
    // (in every thread) when a wait ran out; fin is not run then.
    template <int Q, class F>
    __device__ bool sum(const double (&v)[Q], F fin) {
        set ^= 1u;
        const double a = team_block_sum<Q>(v, sh->red);
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (wid < Q) {
            double* parts = buf->parts[set][wid];
            unsigned long long* total = buf->total[set][wid].half;
            unsigned* n = &buf->arrived[wid].n;
            unsigned target = 0, old = 0;
            if (lane == 0) {
                target = sh->target[wid] + (unsigned)size;
                sh->target[wid] = target;
                asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(parts + rank), "d"(a) : "memory");
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(n) : "memory");
            }
            if (__shfl_sync(0xffffffffu, old + 1u == target, 0)) {
                __syncwarp();   // lane 0 has acquired the others' sums: now every lane may read them
                double s = 0.;
                for (int b = lane; b < size; b += 32) {
                    double p;
                    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(p) : "l"(parts + b) : "memory");
                    s += p;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += team_xor(s, o);
                if (lane == 0) {
                    const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
                    const unsigned long long tag = (unsigned long long)target << 32;
                    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(total), "l"(tag | (bits & 0xffffffffull))
                                 : "memory");
                    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(total + 1), "l"(tag | (bits >> 32))
                                 : "memory");
                    sh->tot[wid] = s;
                }
            } else if (lane == 0) {
                // the total, and with the counter's value (acquired) every
                // store that any block made before it counted itself in
                unsigned long long lo, hi;
                unsigned have;
                int polls = 0;
                bool wait;
                do {
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(lo) : "l"(total) : "memory");
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(hi) : "l"(total + 1) : "memory");
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(have) : "l"(n) : "memory");
                    wait = (unsigned)(lo >> 32) != target || (unsigned)(hi >> 32) != target || (int)(have - target) < 0;
                } while (wait && ++polls < sh->limit);
                if (wait) sh->timeout = 1;
                sh->tot[wid] = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
            }
        }
        if (Q > 1) __syncthreads();   // (one value: thread 0's own warp)
        if (threadIdx.x == 0 && !sh->timeout) fin(sh->tot);
        __syncthreads();
        return sh->timeout == 0;
    }
};

// The blocks of a cluster: block sums go to every block's shared memory and
// the cluster's barrier orders them, with every store before it (1.0 us an
// exchange on 16 blocks of 512 threads, 0.9 on 8, most of it the block's own
// sum).  Two sets, as in a grid team.
struct ClusterTeam {
    TeamShared* sh;
    int rank, size;
    unsigned set;

    // Before the first store to another block's shared memory: the blocks of a
    // cluster are placed together but need not have started together, and the
    // shared memory of one that has not may not be touched.
    __device__ void start() const { barrier(); }
    __device__ void stop() {}
    __device__ static ClusterTeam here(TeamShared* sh) {
        unsigned r, n;
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
        return ClusterTeam{sh, (int)r, (int)n, 0u};
    }
    __device__ void barrier() const {
        if (size == 1) {
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
    }
    // the shared-memory address of p in block b of the cluster
    __device__ static unsigned remote(const void* p, int b) {
        unsigned a;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(b));
        return a;
    }
    // as GridTeam::sum; a hardware barrier does not run out
    template <int Q, class F>
    __device__ bool sum(const double (&v)[Q], F fin) {
        set ^= 1u;
        const double a = team_block_sum<Q>(v, sh->red);
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (wid < Q && lane < size)
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote(&sh->parts[set][wid][rank], lane)), "d"(a)
                         : "memory");
        barrier();
        if (wid == 0) {
            double t[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) {
                t[q] = lane < size ? sh->parts[set][q][lane] : 0.;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) t[q] += team_xor(t[q], o);
            }
            if (lane == 0) fin(t);
        }
        __syncthreads();
        return true;
    }
};

// Row geometry of a stored system: the components' planes are stacked along i
// and wrap inside their component.
struct TeamGeo {
    int n0, n1, n2;     // one component
    int sx, sy;         // strides of i and j
    int off[6];         // step to the neighbour past each face: the wrap, or 0
    unsigned gone;      // faces without a neighbour beyond (bit per face W,E,S,N,B,T)
};
inline TeamGeo team_geo(const GridDev& g) {
    TeamGeo t{};
    t.n0 = g.n[0] / g.ncomp;
    t.n1 = g.n[1];
    t.n2 = g.n[2];
    t.sx = g.n[1] * g.n[2];
    t.sy = g.n[2];
    const int st[3] = {t.sx, t.sy, 1}, n[3] = {t.n0, t.n1, t.n2};
    for (int d = 0; d < 3; d++) {
        t.off[2 * d] = g.periodic[d] ? (n[d] - 1) * st[d] : 0;
        t.off[2 * d + 1] = -t.off[2 * d];
        if (!g.periodic[d]) t.gone |= 3u << (2 * d);
    }
    return t;
}
// bit per face of the cell's grid that the cell touches
__device__ __forceinline__ unsigned team_faces(const TeamGeo& g, int c) {
    const int i = (c / g.sx) % g.n0, rem = c % g.sx, j = rem / g.sy, k = rem - j * g.sy;
    return (i == 0) | (i == g.n0 - 1) << 1 | (j == 0) << 2 | (j == g.n1 - 1) << 3 | (k == 0) << 4 |
           (k == g.n2 - 1) << 5;
}
// Vectors of a team solve (global memory, the iterate's values in r and u)
struct TeamVecs {
    double *x, *rh, *r, *u, *v, *s, *w, *t;
};

// The iterations, from a state that finish_init has set, until it is done:
// the passes K1 .. K5 of dare_march.cuh over this block's cells.  Op gives
//   pass(zf, pre, body): for each of the block's cells, body(c, y, z0, pre(c))
//     with y the operator's row for the operand zf and z0 its own value (pre
//     is called early, so that its loads run beside the operand's);
//   each<U>(body): body(c) for each cell, U of them at a time.
// Returns false when a wait of the team ran out.
// The four SpMV passes are one loop over (a, b, out, coefficient): every
// operand has the form b + coefficient a, and the code of one pass keeps the
// registers of one pass (four copies of it spilled 360 bytes a thread).
template <class Team, class Op>
__device__ bool team_iterations(Team& team, Op& op, const TeamVecs& V, SolverState* st) {
    while (!st->done) {
#pragma unroll 1
        for (int stage = 0; stage < 4; stage++) {
            // (5)-(7): v = Op(r - beta5 u); (8), (9), (11): s = Op(r - alpha1 v);
            // (12)-(14): w = Op(s - beta v); (16)-(20): t = Op(s - alpha w)
            const double* a = stage == 0 ? V.u : stage == 3 ? V.w : V.v;
            const double* b = stage < 2 ? V.r : V.s;
            double* out = stage == 0 ? V.v : stage == 1 ? V.s : stage == 2 ? V.w : V.t;
            const double alpha = st->alpha, alpha1 = st->alpha1, beta = st->beta;
            const double coef = stage & 1 ? -alpha : -beta;
            double dot[5] = {0., 0., 0., 0., 0.};
            op.pass([&](int e) { return coef * a[e] + b[e]; },
                    [&](int c) {
                        return stage < 3 ? V.rh[c] : r_of_16(V.r[c], V.v[c], V.s[c], alpha1, alpha, beta);
                    },
                    [&](int c, double y, double z, double p) {
                        out[c] = y;
                        if (stage < 3) {
                            // (fused as in the initial residual's sum: where Op is the
                            // identity both add the same products, and alpha is 1)
                            dot[0] = fma(y, p, dot[0]);
                        } else {
                            dot[0] += p * z;
                            dot[1] += z * z;
                            dot[2] += z * y;
                            dot[3] += y * y;
                            dot[4] += p * y;
                        }
                    });
            if (stage < 3) {
                const double d1[1] = {dot[0]};
                if (!team.template sum<1>(d1, [&](const double* t) {
                        if (stage == 1)
                            finish_rho(st, t);
                        else
                            finish_gamma(st, t, stage == 0 ? 7 : 14);
                    }))
                    return false;
            } else if (!team.template sum<5>(dot, [&](const double* t) { finish_omega(st, t); })) {
                return false;
            }
            if (st->done) return true;
        }
        const Step5<double> f(st);
        double a2[2] = {0., 0.};
        op.template each<2>([&](int c) {                                // (10), (15), (24), (25)
            double xc = V.x[c], rc = V.r[c], uc = V.u[c];
            f.cell(xc, rc, uc, V.v[c], V.s[c], V.w[c], V.t[c]);
            V.x[c] = xc;
            V.r[c] = rc;
            V.u[c] = uc;
            a2[0] += rc * rc;
            a2[1] += V.rh[c] * rc;
        });
        if (!team.template sum<2>(a2, [&](const double* t) { finish_update(st, t); })) return false;
    }
    return true;
}

}  // namespace dare_gpu
