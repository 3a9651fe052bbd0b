// dare_resident.cu -- the plain FP64 BiCGStab(2) solve of a small system as
// one kernel, a cooperative launch or a single cluster (dare_team.cuh): the
// fold, the iterations and the exit, with CopyTo and the periodic ghosts in a time step.
//
// What bounds a small solve is not its bytes: a 64^3 iteration moves 109 MB
// through L2 but its five kernels, each a launch with a queue of items and a
// pipeline to fill, took 26 us, and the host queued up to 16 iterations before
// it looked at the state, the rest of them empty launches.  Here every block
// keeps its rows of the folded operator in shared memory, the vectors stay in
// L2, an exchange between blocks takes the place of a launch, and the kernel
// ends when the solve does.  A time step, before and after: 64^3 diffusion 376
// -> 167 us, 97 x 61 x 75 TVD 737 -> 360 us, 96 x 80 with two species 364 ->
// 109 us (as one cluster; the solve is 76 of it).  The solve alone takes 140 us
// at 64^3, 293 for 97 x 61 x 75.  What is left of a pass with its exchange (64^3, 6 us): forming the
// operand 1.8 us, the rows 1 us, the block's sum 0.4 us, publishing it 1.1 us
// and the total coming back 1.9 us, all of them L2 round trips of ~0.5 us.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "dare_team.cuh"

using namespace dare_gpu;

namespace dare_gpu {

struct ResidentArgs {
    TeamGeo geo;
    GridDev grid;              // one component (the field's ghosts)
    int ncell, chunk;          // all components; cells of a block
    const double *diag, *b;    // 7 diagonals of ncell each, rhs
    double *invd, *field;      // field: level 0 to write at the exit (null: none)
    TeamVecs v;
    double tol;
    int max_it, tol_relative, want_residual;
    TeamBuffer* buf;
    int polls, quitter;            // limit of a block's waits; the block whose limit is 0 (-1: none)
    SolverState *st, *st_host;     // results (device copy, pinned host copy)
    int* gave_up;                  // pinned host word that a block sets when a wait of it ran out
};

// 1024 threads and one block per SM: 64 registers each, and 32 warps to hide
// the L2 latency of one another.
constexpr int kResidentThreads = 1024;

// The rows of this block in shared memory: NC coefficients of m cells (stride
// `stride`), the faces each cell touches, and a tile for the operand on the
// block's cells and the rows before and after them, where the j and k
// neighbours are.  A block's cells are a run in memory, usually shorter than a
// plane, so the i neighbours have no second reader here: each thread forms
// its own cells' from global memory.  CPT cells a thread, all their loads in
// flight before the barrier: a 64^3 pass takes 2.6 us (operand formed at all 7
// points from L1 3.1 us), an 82^3 pass 4.8 us (6.6).
template <bool UNIT, int CPT>
struct ResidentOp {
    const TeamGeo& geo;
    double *coef, *tile;
    unsigned char* faces;
    int ncell, stride, m, c0;

    // the thread's first cell, opaque to the compiler: otherwise it keeps the
    // addresses of every cell from one pass to the next, in spilled registers
    __device__ __forceinline__ int first() const {
        int t = threadIdx.x;
        asm volatile("" : "+r"(t));
        return t;
    }
    __device__ __forceinline__ bool gone(unsigned f, int q) const { return (f & geo.gone) >> q & 1u; }
    template <class ZF, class Pre, class Body>
    __device__ __forceinline__ void pass(ZF zf, Pre pre, Body body) {
        constexpr int nt = kResidentThreads;
        const int tid = first(), sy = geo.sy;
        double zw[CPT], ze[CPT], p[CPT];
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            const int lc = tid + q * nt, c = c0 + lc;
            if (lc < m) {
                const unsigned f = faces[lc];
                const double z = zf(c);
                const double w = zf(c + (f & 1u ? geo.off[0] : -geo.sx)), e = zf(c + (f & 2u ? geo.off[1] : geo.sx));
                p[q] = pre(c);
                zw[q] = gone(f, 0) ? 0. : w;
                ze[q] = gone(f, 1) ? 0. : e;
                tile[sy + lc] = z;
            }
        }
        for (int h = tid; h < 2 * sy; h += nt) {
            const int lc = h < sy ? h - sy : m + h - sy, c = c0 + lc;
            tile[sy + lc] = c >= 0 && c < ncell ? zf(c) : 0.;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            const int lc = tid + q * nt, c = c0 + lc;
            if (lc < m) {
                const unsigned f = faces[lc];
                const double *t = tile + sy + lc, *a = coef + lc;
                // past a periodic j face the neighbour is n1 - 1 rows away,
                // past a k face n2 - 1 cells: inside the tile
                const double s = gone(f, 2) ? 0. : f & 4u ? zf(c + geo.off[2]) : t[-sy];
                const double n = gone(f, 3) ? 0. : f & 8u ? zf(c + geo.off[3]) : t[sy];
                const double b = gone(f, 4) ? 0. : t[f & 16u ? geo.off[4] : -1];
                const double u = gone(f, 5) ? 0. : t[f & 32u ? geo.off[5] : 1];
                double y = UNIT ? t[0] : a[6 * stride] * t[0];
                y += a[0] * zw[q];
                y += a[stride] * ze[q];
                y += a[2 * stride] * s;
                y += a[3 * stride] * n;
                y += a[4 * stride] * b;
                y += a[5 * stride] * u;
                body(c, y, t[0], p[q]);
            }
        }
    }
    template <int U, class Body>
    __device__ __forceinline__ void each(Body body) {
#pragma unroll U
        for (int lc = first(); lc < m; lc += kResidentThreads) body(c0 + lc);
    }
    // f at the six neighbours of own cell c, zero where there is none
    template <class F>
    __device__ __forceinline__ void neighbours(int c, F f, double (&z)[6]) const {
        const int step[6] = {-geo.sx, geo.sx, -geo.sy, geo.sy, -1, 1};
        const unsigned at = faces[c - c0];
#pragma unroll
        for (int q = 0; q < 6; q++) z[q] = gone(at, q) ? 0. : f(c + (at >> q & 1u ? geo.off[q] : step[q]));
    }
};

// CLUSTER: the blocks are one cluster, otherwise those of a cooperative launch
template <bool UNIT, int CPT, bool CLUSTER>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident(ResidentArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TeamShared sh;
    __shared__ SolverState st_s;
    SolverState* st = &st_s;
    const int tid = threadIdx.x;
    constexpr int NC = NCoef<UNIT>::value;
    const int64_t n = A.ncell;
    const int ch = A.chunk, c0 = blockIdx.x * ch, m = max(0, min(ch, A.ncell - c0));
    double* smem = reinterpret_cast<double*>(smem_raw);
    ResidentOp<UNIT, CPT> op{A.geo, smem,      smem + (size_t)NC * ch,
                             reinterpret_cast<unsigned char*>(smem + (size_t)(NC + 1) * ch + 2 * A.geo.sy),
                             A.ncell, ch, m, c0};
    const auto make_team = [&]() {
        if constexpr (CLUSTER)
            return ClusterTeam::here(&sh);
        else
            return GridTeam{A.buf, &sh, (int)blockIdx.x, (int)gridDim.x, (int)blockIdx.x == A.quitter ? 0 : A.polls,
                            0u};
    };
    auto team = make_team();
    team.start();
    if (tid == 0) {
        SolverState z{};
        z.tol = A.tol;
        z.max_it = A.max_it;
        z.tol_relative = A.tol_relative;
        *st = z;
    }
    op.template each<1>([&](int c) {
        op.faces[c - c0] = (unsigned char)team_faces(A.geo, c);
        if (UNIT) A.invd[c] = 1. / A.diag[c];
    });
    bool ok = true;
    const double none[1] = {0.};
    __syncthreads();
    if (UNIT) ok = team.template sum<1>(none, [](const double*) {});   // invd of every block
    // Ahat = A D^-1 (columns scaled) into shared memory; r = b - Ahat y,
    // r_hat_0 = r, u = 0
    if (ok) {
        op.template each<1>([&](int c) {
            double iv[6];
            if (UNIT) op.neighbours(c, [&](int e) { return A.invd[e]; }, iv);
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const double a = A.diag[(q + 1) * n + c];
                op.coef[q * ch + c - c0] = UNIT ? a * iv[q] : a;
            }
            if (!UNIT) op.coef[6 * ch + c - c0] = A.diag[c];
        });
        double a2[2] = {0., 0.};
        op.pass([&](int e) { return A.v.x[e]; }, [&](int c) { return A.b[c]; },
                [&](int c, double y, double, double bc) {
                    const double rr = bc - y;
                    A.v.r[c] = rr;
                    A.v.rh[c] = rr;
                    A.v.u[c] = 0.;
                    a2[0] = fma(rr, rr, a2[0]);
                    a2[1] += bc * bc;
                });
        ok = team.template sum<2>(a2, [&](const double* t) { finish_init(st, t); }) && team_iterations(team, op, A.v, st);
    }
    if (ok) {
        // the exit: step (10) when the solve stopped between it and the last
        // pass, x = D^-1 y, CopyTo and the periodic face ghosts (each written
        // by the internal cell it images, as k_solution_to_field does)
        const bool pend = step10_pending_state(st->status, st->step);
        const double alpha1 = st->alpha1, beta5 = st->beta5;
        const GridDev& g = A.grid;
        op.template each<1>([&](int c) {
            double xc = A.v.x[c];
            if (pend) {
                const double u5 = A.v.r[c] - beta5 * A.v.u[c];
                xc = alpha1 * u5 + xc;
            }
            if (UNIT) xc = A.invd[c] * xc;
            if (UNIT || pend) A.v.x[c] = xc;
            if (!A.field) return;
            const int ia = c / A.geo.sx, rem = c - ia * A.geo.sx, j = rem / A.geo.sy, k = rem - j * A.geo.sy;
            const int comp = ia / A.geo.n0;
            double* phi = A.field + (size_t)comp * g.ncell_ghosted;
            const int q[3] = {ia - comp * A.geo.n0, j, k};
            const int ind[3] = {q[0] + g.og[0], q[1] + g.og[1], q[2] + g.og[2]};
            phi[((int64_t)ind[0] * g.gn[1] + ind[1]) * g.gn[2] + ind[2]] = xc;
            for (int d = 0; d < g.dim; d++) {
                if (!g.periodic[d]) continue;
                int p[3] = {ind[0], ind[1], ind[2]};
                if (q[d] < g.ng) {
                    p[d] = g.og[d] + g.n[d] + q[d];
                    phi[((int64_t)p[0] * g.gn[1] + p[1]) * g.gn[2] + p[2]] = xc;
                }
                if (q[d] >= g.n[d] - g.ng) {
                    p[d] = q[d] - g.n[d] + g.ng;
                    phi[((int64_t)p[0] * g.gn[1] + p[1]) * g.gn[2] + p[2]] = xc;
                }
            }
        });
        if (A.want_residual) {   // ||b - A x||_2 with the assembled rows
            ok = team.template sum<1>(none, [](const double*) {});
            double a1[1] = {0.};
            if (ok) {
                op.template each<1>([&](int c) {
                    double z[7], p[7], zn[6];
                    op.neighbours(c, [&](int e) { return A.v.x[e]; }, zn);
                    z[0] = A.v.x[c];
                    p[6] = A.diag[c];
#pragma unroll
                    for (int q = 0; q < 6; q++) {
                        z[q + 1] = zn[q];
                        p[q] = A.diag[(q + 1) * n + c];
                    }
                    const double r = A.b[c] - apply_pre<double, false>(p, z);
                    a1[0] += r * r;
                });
                ok = team.template sum<1>(a1, [&](const double* t) { st->tres = sqrt(t[0]); });
            }
        }
    }
    // Block 0 reports the state, and every block whose wait ran out says so
    // itself: at the last exchange block 0 may get the total that another one
    // has given up waiting for, with its cells unfinished.
    team.stop();
    if (!ok && tid == 0) *A.gave_up = 1;
    if (blockIdx.x == 0 && tid == 0) {
        *A.st = *st;
        *A.st_host = *st;
    }
}

constexpr int kResidentCells = 4;   // most cells a thread
// Measured solves, cluster / device: 24^3 43 / 59 us, 32^3 58 / 60, 36^3 94 / 83;
// two species on 90^2 76 / 103, 120^2 113 / 128, 160^2 211 / 168
constexpr int64_t kClusterCells = 1 << 15;
constexpr size_t kResidentSmem = 227 * 1024 - sizeof(TeamShared) - sizeof(SolverState) - 1024;
static size_t resident_smem(bool unit, int chunk, int sy) {
    return ((size_t)chunk * (unit ? 7 : 8) + 2 * (size_t)sy) * sizeof(double) + chunk;
}

template <bool UNIT, bool CLUSTER>
static const void* resident_kernel_t(int chunk) {
    switch ((chunk + kResidentThreads - 1) / kResidentThreads) {
    case 1: return (const void*)k_resident<UNIT, 1, CLUSTER>;
    case 2: return (const void*)k_resident<UNIT, 2, CLUSTER>;
    case 3: return (const void*)k_resident<UNIT, 3, CLUSTER>;
    default: return (const void*)k_resident<UNIT, kResidentCells, CLUSTER>;
    }
}
static const void* resident_kernel(bool unit, const ResidentPlan& P) {
    if (unit) return P.cluster ? resident_kernel_t<true, true>(P.chunk) : resident_kernel_t<true, false>(P.chunk);
    return P.cluster ? resident_kernel_t<false, true>(P.chunk) : resident_kernel_t<false, false>(P.chunk);
}
static cudaLaunchConfig_t resident_config(const dare_ctx* ctx, const ResidentPlan& P, size_t smem,
                                          cudaLaunchAttribute* at) {
    if (P.cluster) {
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = (unsigned)P.blocks;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
    } else {
        at->id = cudaLaunchAttributeCooperative;
        at->val.cooperative = 1;
    }
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(P.blocks);
    c.blockDim = dim3(kResidentThreads);
    c.dynamicSmemBytes = smem;
    c.stream = ctx->stream;
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}
// (the kernels' limit is the most that any system takes, not one system's need:
// it belongs to the kernel, and other threads launch it for other systems)
static cudaError_t resident_limits(const void* k, bool cluster) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResidentSmem);
    if (e == cudaSuccess && cluster) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// A team of at most `most` blocks: as many as have a cell for each of half
// their threads (below that an SM more does not shorten a pass).  False when a
// block's rows do not fit its shared memory, or the device (or this process's
// share of it) cannot hold the team's blocks at the same time.
static bool resident_team(const dare_ctx* ctx, const GridDev& g, bool unit, bool cluster, int64_t most,
                          ResidentPlan& P) {
    const int64_t n = g.ncell;
    if (most < 1 || n > most * kResidentThreads * kResidentCells || g.n[2] > (1 << 15)) return false;
    const int64_t want = std::min(most, (n + kResidentThreads / 2 - 1) / (kResidentThreads / 2));
    const int64_t ch = ((n + want - 1) / want + 31) / 32 * 32;
    const size_t smem = resident_smem(unit, (int)ch, g.n[2]);
    if (ch > kResidentThreads * kResidentCells || smem > kResidentSmem) return false;
    P.cluster = cluster;
    P.chunk = (int)ch;
    P.blocks = (int)((n + ch - 1) / ch);
    const void* k = resident_kernel(unit, P);
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t c = resident_config(ctx, P, smem, at);
    int fit = 0;
    cudaError_t e = resident_limits(k, cluster);
    if (e == cudaSuccess)
        e = cluster ? cudaOccupancyMaxActiveClusters(&fit, k, &c)
                    : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, kResidentThreads, smem);
    if (e != cudaSuccess) cudaGetLastError();
    if (e == cudaSuccess && (cluster ? fit >= 1 : (int64_t)fit * ctx->num_sms >= P.blocks)) return true;
    P.blocks = 0;
    return false;
}

// The team that solves a system in one launch, found at its first solve;
// blocks = 0 when there is none, and the marching kernels solve it (beyond that
// size they are the faster path, their vectors no longer stay in L2 either).
// Up to kClusterCells cells one cluster, whose exchanges take 1 us where the
// device's take 3; beyond that, or without room for the cluster, blocks of the
// whole device, whose passes are shorter.
const ResidentPlan& resident_plan(const dare_ctx* ctx, const GridDev& g, bool unit, dare_solver_ws* ws) {
    ResidentPlan& P = ws->resident[unit];
    if (P.known && P.most_cluster == ctx->team_cluster && P.most_grid == ctx->team_grid) return P;
    P = ResidentPlan{};
    P.most_cluster = ctx->team_cluster;
    P.most_grid = ctx->team_grid;
    const auto at_most = [](int blocks, int limit) { return limit < 0 ? blocks : std::min(blocks, limit); };
    const bool found = (g.ncell <= kClusterCells &&
                        resident_team(ctx, g, unit, true, at_most(kClusterMaxBlocks, P.most_cluster), P)) ||
                       resident_team(ctx, g, unit, false, at_most(std::min(ctx->num_sms, kTeamMaxBlocks), P.most_grid), P);
    if (!found) P.blocks = 0;
    P.known = true;
    return P;
}

// The whole solve of system s in one launch: x (and field level 0 when given)
// and the final state, in ws->st_host once the stream is synchronized.
int launch_resident(dare_system* s, const dare_solver_params* p, const VecsT<double>& vs, const ResidentPlan& P,
                    double* field) {
    dare_ctx* ctx = s->grid->ctx;
    dare_solver_ws* ws = s->ws;
    const GridDev& g = s->sdev;
    ResidentArgs a{};
    a.geo = team_geo(g);
    a.grid = s->grid->dev;
    a.ncell = (int)g.ncell;
    a.chunk = P.chunk;
    a.diag = s->diag;
    a.b = s->rhs;
    a.invd = ws->invd;
    a.field = field;
    a.v = TeamVecs{vs.x, vs.rh, vs.r, vs.u, vs.v, vs.s, vs.w, vs.t};
    a.tol = p->tol;
    a.max_it = p->max_it;
    a.tol_relative = p->tol_relative;
    a.want_residual = p->compute_true_residual;
    a.buf = static_cast<TeamBuffer*>(ws->team_buf);
    a.polls = ctx->team_polls > 0 ? ctx->team_polls : kTeamPolls;
    a.quitter = ctx->debug_quitter;
    ctx->debug_quitter = -1;
    a.st = ws->st;
    a.st_host = ws->st_host;
    a.gave_up = ws->gave_up;
    *ws->gave_up = 0;   // (no kernel of this workspace is running)
    const bool unit = p->precond == DARE_PREC_JACOBI;
    const void* k = resident_kernel(unit, P);
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t c = resident_config(ctx, P, resident_smem(unit, P.chunk, a.geo.sy), at);
    void* args[] = {&a};
    DARE_CUDA(ctx, resident_limits(k, P.cluster));
    DARE_CUDA(ctx, cudaLaunchKernelExC(&c, k, args));
    DARE_LAUNCHED(ctx);
    return DARE_OK;
}

}  // namespace dare_gpu
