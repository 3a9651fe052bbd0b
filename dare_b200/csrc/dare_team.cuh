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

constexpr int kTeamMaxBlocks = 160;   // blocks of a grid team (packets of one exchange)
constexpr int kTeamEpoch = 2 * kMaxQ * kTeamMaxBlocks * 2;   // word of a grid team's buffer: its last exchange
constexpr size_t kTeamBytes = (kTeamEpoch + 1) * sizeof(unsigned long long);

// Block part of a sum: afterwards warp q (q < Q) holds the block's sum of
// value q in every lane.  The barrier inside also orders every store of the
// block before what those warps do next.
template <int Q>
__device__ __forceinline__ double team_block_sum(double (&v)[Q], double* red /* [32 * kMaxQ] */) {
#pragma unroll
    for (int q = 0; q < Q; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < Q; q++) red[q * 32 + wid] = v[q];
    }
    __syncthreads();
    double a = 0.;
    if (wid < Q) {
        a = lane < ((int)blockDim.x >> 5) ? red[wid * 32 + lane] : 0.;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    }
    return a;
}

// Shared-memory scratch of a team's exchanges.
struct TeamShared {
    double red[32 * kMaxQ];
    double parts[kMaxQ * kTeamMaxBlocks];   // cluster teams: [2][kMaxQ][16], written by the peers
    int timeout;
};

// The blocks of a cooperative launch.  Each exchange, a block publishes one
// 16-byte packet per value: the double's two halves, each beside the
// exchange's number, so that a reader that sees the number in both words has
// the value (8-byte stores are single) and needs no separate flag.  Every
// block polls the packets of all blocks: one store and one load latency,
// without atomics.  Packets alternate between two sets: a block can be one
// exchange ahead of another at most, which still reads the other set.
// Every wait ends: after kTeamPolls polls the block gives up, and so do the
// blocks that wait for it.
constexpr int kTeamPolls = 1 << 22;
struct GridTeam {
    unsigned long long* packets;   // [2][kMaxQ][size][2]
    TeamShared* sh;
    int rank, size;
    unsigned epoch;                // number of the last exchange

    // Totals of Q values in thread 0 (tot), after a barrier of the team.
    // False when a wait ran out.
    template <int Q>
    __device__ bool sum(double (&v)[Q], double (&tot)[Q]) {
        epoch++;
        const double a = team_block_sum<Q>(v, sh->red);
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        unsigned long long* set = packets + (size_t)(epoch & 1u) * kMaxQ * size * 2;
        const unsigned long long tag = (unsigned long long)epoch << 32;
        if (wid < Q && lane == 0) {
            const unsigned long long bits = (unsigned long long)__double_as_longlong(a);
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(set + 2 * ((size_t)wid * size + rank)),
                         "l"(tag | (bits & 0xffffffffull)), "l"(tag | (bits >> 32))
                         : "memory");
        }
        bool mine = false;
        for (int p = threadIdx.x; p < Q * size; p += blockDim.x) {
            unsigned long long lo, hi;
            int polls = 0;
            do {
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(set + 2 * (size_t)p)
                             : "memory");
            } while (((lo ^ tag) >> 32 || (hi ^ tag) >> 32) && ++polls < kTeamPolls);
            if (polls >= kTeamPolls) sh->timeout = 1;
            sh->parts[p] = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
            mine = true;
        }
        if (mine) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        __syncthreads();
        if (wid == 0) {
#pragma unroll
            for (int q = 0; q < Q; q++) {
                double s = 0.;
                for (int b = lane; b < size; b += 32) s += sh->parts[q * size + b];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                tot[q] = s;
            }
        }
        return sh->timeout == 0;
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
// the operand zf at the 7 points of cell c, a removed neighbour's value zero
template <class F>
__device__ __forceinline__ void team_points(const TeamGeo& g, int c, unsigned f, F zf, double (&z)[7]) {
    const int step[6] = {-g.sx, g.sx, -g.sy, g.sy, -1, 1};
    z[0] = zf(c);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const bool at = f >> q & 1u;
        const double a = zf(c + (at ? g.off[q] : step[q]));
        z[q + 1] = at && (g.gone >> q & 1u) ? 0. : a;
    }
}

// Vectors of a team solve (global memory, the iterate's values in r and u)
struct TeamVecs {
    double *x, *rh, *r, *u, *v, *s, *w, *t;
};

// The iterations, from a state that finish_init has set, until it is done:
// the passes K1 .. K5 of dare_march.cuh over this block's cells.  Op gives
// m (cells of the block), c0 (the first) and
//   row(lc, c, zf, z0): the operator's row for operand zf, its own value in z0.
// Returns false when a wait of the team ran out.
template <class Team, class Op>
__device__ bool team_iterations(Team& team, const Op& op, const TeamVecs& V, SolverState* st) {
    const int tid = threadIdx.x, nt = blockDim.x;
    while (!st->done) {
        double a1[1] = {0.}, t1[1] = {0.};
        const double beta5 = st->beta;
        for (int lc = tid; lc < op.m; lc += nt) {                       // (5)-(7)
            const int c = op.c0 + lc;
            double z0;
            const double vc = op.row(lc, c, [&](int e) { return V.r[e] - beta5 * V.u[e]; }, z0);
            V.v[c] = vc;
            a1[0] += vc * V.rh[c];
        }
        if (!team.template sum<1>(a1, t1)) return false;
        if (tid == 0) finish_gamma(st, t1, 7);
        __syncthreads();
        if (st->done) break;
        const double alpha1 = st->alpha;
        a1[0] = 0.;
        for (int lc = tid; lc < op.m; lc += nt) {                       // (8), (9), (11)
            const int c = op.c0 + lc;
            double z0;
            const double sc = op.row(lc, c, [&](int e) { return -alpha1 * V.v[e] + V.r[e]; }, z0);
            V.s[c] = sc;
            a1[0] += V.rh[c] * sc;
        }
        if (!team.template sum<1>(a1, t1)) return false;
        if (tid == 0) finish_rho(st, t1);
        __syncthreads();
        const double beta = st->beta;
        a1[0] = 0.;
        for (int lc = tid; lc < op.m; lc += nt) {                       // (12)-(14)
            const int c = op.c0 + lc;
            double z0;
            const double wc = op.row(lc, c, [&](int e) { return V.s[e] - beta * V.v[e]; }, z0);
            V.w[c] = wc;
            a1[0] += wc * V.rh[c];
        }
        if (!team.template sum<1>(a1, t1)) return false;
        if (tid == 0) finish_gamma(st, t1, 14);
        __syncthreads();
        if (st->done) break;
        const double alpha = st->alpha;
        double a5[5] = {0., 0., 0., 0., 0.}, t5[5] = {0., 0., 0., 0., 0.};
        for (int lc = tid; lc < op.m; lc += nt) {                       // (16)-(20)
            const int c = op.c0 + lc;
            double ds;
            const double dt = op.row(lc, c, [&](int e) { return -alpha * V.w[e] + V.s[e]; }, ds);
            V.t[c] = dt;
            const double dr = r_of_16(V.r[c], V.v[c], V.s[c], alpha1, alpha, beta);
            a5[0] += dr * ds;
            a5[1] += ds * ds;
            a5[2] += ds * dt;
            a5[3] += dt * dt;
            a5[4] += dr * dt;
        }
        if (!team.template sum<5>(a5, t5)) return false;
        if (tid == 0) finish_omega(st, t5);
        __syncthreads();
        if (st->done) break;
        const Step5<double> f(st);
        double a2[2] = {0., 0.}, t2[2] = {0., 0.};
        for (int lc = tid; lc < op.m; lc += nt) {                       // (10), (15), (24), (25)
            const int c = op.c0 + lc;
            double xc = V.x[c], rc = V.r[c], uc = V.u[c];
            f.cell(xc, rc, uc, V.v[c], V.s[c], V.w[c], V.t[c]);
            V.x[c] = xc;
            V.r[c] = rc;
            V.u[c] = uc;
            a2[0] += rc * rc;
            a2[1] += V.rh[c] * rc;
        }
        if (!team.template sum<2>(a2, t2)) return false;
        if (tid == 0) finish_update(st, t2);
        __syncthreads();
    }
    return true;
}

}  // namespace dare_gpu
