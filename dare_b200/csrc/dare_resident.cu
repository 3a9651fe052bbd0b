// dare_resident.cu -- the plain FP64 BiCGStab(2) solve of a small system as
// one cooperative kernel (dare_team.cuh): the fold, the iterations and the
// exit, with CopyTo and the periodic ghosts in a time step.
//
// What bounds a small solve is not its bytes: a 64^3 iteration moves 109 MB
// through L2 but its five kernels, each a launch with a queue of items and a
// pipeline to fill, took 26 us, and the host queued up to 16 iterations before
// it looked at the state, the rest of them empty launches.  Here every block
// keeps its rows of the folded operator in shared memory, the vectors stay in
// L2, an exchange between blocks takes the place of a launch, and the kernel
// ends when the solve does.
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
    unsigned long long* packets;   // exchange packets, then the number of the last exchange (kTeamEpoch)
    SolverState *st, *st_host;     // results (device copy, pinned host copy)
};

// Rows of this block in shared memory: NC coefficients of m cells (stride
// `chunk`), and the faces each cell touches.
template <bool UNIT>
struct ResidentOp {
    TeamGeo geo;
    const double* coef;
    const unsigned char* faces;
    int stride, m, c0;
    template <class F>
    __device__ __forceinline__ double row(int lc, int c, F zf, double& z0) const {
        double z[7];
        team_points(geo, c, faces[lc], zf, z);
        z0 = z[0];
        double y = UNIT ? z[0] : coef[6 * stride + lc] * z[0];
#pragma unroll
        for (int q = 0; q < 6; q++) y += coef[q * stride + lc] * z[q + 1];
        return y;
    }
};

// 1024 threads and one block per SM: 64 registers each, enough for one cell's
// loads in flight, and 32 warps hide the L2 latency of the others.
constexpr int kResidentThreads = 1024;

template <bool UNIT>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident(ResidentArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TeamShared sh;
    __shared__ SolverState st_s;
    SolverState* st = &st_s;
    const int tid = threadIdx.x, nt = blockDim.x;
    constexpr int NC = NCoef<UNIT>::value;
    double* coef = reinterpret_cast<double*>(smem_raw);
    unsigned char* faces = smem_raw + (size_t)NC * A.chunk * sizeof(double);
    const int c0 = blockIdx.x * A.chunk;
    const int m = max(0, min(A.chunk, A.ncell - c0));
    const int64_t n = A.ncell;
    GridTeam team{A.packets, &sh, (int)blockIdx.x, (int)gridDim.x, (unsigned)A.packets[kTeamEpoch]};
    if (tid == 0) {
        sh.timeout = 0;
        SolverState z{};
        z.tol = A.tol;
        z.max_it = A.max_it;
        z.tol_relative = A.tol_relative;
        *st = z;
    }
    for (int lc = tid; lc < m; lc += nt) {
        faces[lc] = (unsigned char)team_faces(A.geo, c0 + lc);
        if (UNIT) A.invd[c0 + lc] = 1. / A.diag[c0 + lc];
    }
    bool ok = true;
    double none[1] = {0.}, dummy[1];
    if (UNIT) ok = team.sum<1>(none, dummy);   // invd of every block
    else __syncthreads();
    // Ahat = A D^-1 (columns scaled) into shared memory; r = b - Ahat y,
    // r_hat_0 = r, u = 0
    double a2[2] = {0., 0.}, t2[2] = {0., 0.};
    if (ok) {
        const ResidentOp<UNIT> op{A.geo, coef, faces, A.chunk, m, c0};
        for (int lc = tid; lc < m; lc += nt) {
            const int c = c0 + lc;
            if constexpr (UNIT) {
                double iv[7];
                team_points(A.geo, c, faces[lc], [&](int e) { return A.invd[e]; }, iv);
#pragma unroll
                for (int q = 0; q < 6; q++) coef[q * A.chunk + lc] = A.diag[(q + 1) * n + c] * iv[q + 1];
            } else {
#pragma unroll
                for (int q = 0; q < 6; q++) coef[q * A.chunk + lc] = A.diag[(q + 1) * n + c];
                coef[6 * A.chunk + lc] = A.diag[c];
            }
            double y0;
            const double yy = op.row(lc, c, [&](int e) { return A.v.x[e]; }, y0);
            const double bc = A.b[c], rr = bc - yy;
            A.v.r[c] = rr;
            A.v.rh[c] = rr;
            A.v.u[c] = 0.;
            a2[0] += rr * rr;
            a2[1] += bc * bc;
        }
        ok = team.sum<2>(a2, t2);
        if (ok && tid == 0) finish_init(st, t2);
        __syncthreads();
        ok = ok && team_iterations(team, op, A.v, st);
    }
    if (ok) {
        // the exit: step (10) when the solve stopped between it and the last
        // pass, x = D^-1 y, CopyTo and the periodic face ghosts (each written
        // by the internal cell it images, as k_solution_to_field does)
        const bool pend = step10_pending_state(st->status, st->step);
        const double alpha1 = st->alpha1, beta5 = st->beta5;
        const GridDev& g = A.grid;
        for (int lc = tid; lc < m; lc += nt) {
            const int c = c0 + lc;
            double xc = A.v.x[c];
            if (pend) {
                const double u5 = A.v.r[c] - beta5 * A.v.u[c];
                xc = alpha1 * u5 + xc;
            }
            if (UNIT) xc = A.invd[c] * xc;
            if (UNIT || pend) A.v.x[c] = xc;
            if (!A.field) continue;
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
        }
        if (A.want_residual) {   // ||b - A x||_2 with the assembled rows
            ok = team.sum<1>(none, dummy);
            double a1[1] = {0.}, t1[1] = {0.};
            if (ok) {
                for (int lc = tid; lc < m; lc += nt) {
                    const int c = c0 + lc;
                    double z[7];
                    team_points(A.geo, c, faces[lc], [&](int e) { return A.v.x[e]; }, z);
                    double y = A.diag[c] * z[0];
#pragma unroll
                    for (int q = 0; q < 6; q++) y += A.diag[(q + 1) * n + c] * z[q + 1];
                    const double r = A.b[c] - y;
                    a1[0] += r * r;
                }
                ok = team.sum<1>(a1, t1);
            }
            if (tid == 0) st->tres = sqrt(t1[0]);
        }
    }
    // a block that gave up leaves `done` 0 in its copy; block 0 reports
    if (blockIdx.x == 0 && tid == 0) {
        if (!ok) st->done = 0;
        A.packets[kTeamEpoch] = team.epoch;   // every block read it before the first exchange
        *A.st = *st;
        *A.st_host = *st;
    }
}

// The team's shape for a system, or false when a block's rows do not fit its
// shared memory: beyond that the marching kernels are the faster path (their
// vectors no longer stay in L2 either).
static size_t resident_smem(bool unit, int chunk) {
    return (size_t)chunk * ((unit ? 6 : 7) * sizeof(double) + 1);
}
bool resident_shape(const dare_ctx* ctx, int64_t n, bool unit, int* blocks, int* chunk) {
    constexpr size_t kMost = 227 * 1024 - sizeof(TeamShared) - sizeof(SolverState) - 1024;
    const int nb = ctx->num_sms < kTeamMaxBlocks ? ctx->num_sms : kTeamMaxBlocks;
    if (n > (int64_t)nb * 8192) return false;
    // as many blocks as have a cell for each of half their threads: below
    // that an SM more does not shorten a pass
    int64_t want = (n + kResidentThreads / 2 - 1) / (kResidentThreads / 2);
    if (want > nb) want = nb;
    int64_t ch = (n + want - 1) / want;
    ch = (ch + 31) / 32 * 32;
    if (resident_smem(unit, (int)ch) > kMost) return false;
    *chunk = (int)ch;
    *blocks = (int)((n + ch - 1) / ch);
    return true;
}

template <bool UNIT>
static int launch_resident_t(dare_ctx* ctx, ResidentArgs& a, int blocks) {
    const size_t smem = resident_smem(UNIT, a.chunk);
    DARE_CUDA(ctx, cudaFuncSetAttribute(k_resident<UNIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    void* args[] = {&a};
    DARE_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)k_resident<UNIT>, dim3(blocks), dim3(kResidentThreads), args,
                                               smem, ctx->stream));
    DARE_LAUNCHED(ctx);
    return DARE_OK;
}

// The whole solve of system s in one launch: x (and field level 0 when given)
// and the final state, in ws->st_host once the stream is synchronized.
int launch_resident(dare_system* s, const dare_solver_params* p, const VecsT<double>& vs, int blocks, int chunk,
                    double* field) {
    dare_ctx* ctx = s->grid->ctx;
    dare_solver_ws* ws = s->ws;
    const GridDev& g = s->sdev;
    ResidentArgs a{};
    a.geo = team_geo(g);
    a.grid = s->grid->dev;
    a.ncell = (int)g.ncell;
    a.chunk = chunk;
    a.diag = s->diag;
    a.b = s->rhs;
    a.invd = ws->invd;
    a.field = field;
    a.v = TeamVecs{vs.x, vs.rh, vs.r, vs.u, vs.v, vs.s, vs.w, vs.t};
    a.tol = p->tol;
    a.max_it = p->max_it;
    a.tol_relative = p->tol_relative;
    a.want_residual = p->compute_true_residual;
    a.packets = ws->packets;
    a.st = ws->st;
    a.st_host = ws->st_host;
    return p->precond == DARE_PREC_JACOBI ? launch_resident_t<true>(ctx, a, blocks)
                                          : launch_resident_t<false>(ctx, a, blocks);
}

}  // namespace dare_gpu
