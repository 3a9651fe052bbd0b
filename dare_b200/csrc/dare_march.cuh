// dare_march.cuh -- device side of the BiCGStab(2) kernels: the scalar
// recurrences of BiCGStab2.inl, the fused stencil functors and the
// plane-marching stencil kernel they run in.
//
// The marching kernel is persistent: one grid of (blocks per SM x SMs)
// blocks pulls equal work items -- a (j,k) tile and a run of i-planes -- from
// a device queue.  Inside an item the block walks along i.  Every plane is
// staged in shared memory by asynchronous copies (cp.async): the inputs of the
// fused SpMV operand with a one-cell j/k halo, and the per-cell streams of the
// centre step (coefficients, vectors).  A ring of stages keeps the
// copies of the next planes in flight while plane i computes, so HBM
// latency hides behind the arithmetic without holding data in registers.
// Dot-product partials are kept per item and summed in item order by the
// last item, so results do not depend on which block took which item.
#pragma once

#include <type_traits>

#include "dare_bicgstab2.cuh"

namespace dare_gpu {

// ---------------------------------------------------------------------------
// scalar recurrences, run by thread 0 of the block that finishes last
// ---------------------------------------------------------------------------
__device__ __forceinline__ void finish(SolverState* st, int status, int step) {
    st->status = status;
    st->step = step;
    st->done = 1;
}

// Loop-top bookkeeping of the reference: `if (k > max_iteration) break;`,
// step (3) and step (4) given rho1 = <r_hat_0, r>.
__device__ inline void begin_iteration(SolverState* st, double rho1) {
    if (st->k > st->max_it) {
        finish(st, ST_MAXIT, 0);
        return;
    }
    st->rho0 = -st->omega2 * st->rho0;                       // (3)
    if (st->rho0 == 0.0) {
        finish(st, ST_BREAKDOWN, 3);
        return;
    }
    st->rho1 = rho1;                                         // (4)
    st->beta = st->alpha * st->rho1 / st->rho0;
    st->beta5 = st->beta;                                    // step (5)'s, used again in the last kernel
    st->rho0 = st->rho1;
    if (st->rho0 == 0.0) finish(st, ST_BREAKDOWN, 4);
}

__device__ inline void finish_init(SolverState* st, const double* tot) {
    st->bnorm2 = tot[1];
    if (st->tol_relative) st->tol = st->tol * sqrt(tot[1]);
    st->rnorm0 = sqrt(tot[0]);
    st->rnorm = st->rnorm0;
    st->alpha = 0.;                                           // BiCGStab2.inl:182
    st->rho0 = st->omega1 = st->omega2 = 1.;                 // (1)
    st->k = 0;
    if (st->rnorm0 < st->tol) {                               // initial guess converged
        finish(st, ST_CONVERGED, 0);
        return;
    }
    if (isnan(st->rnorm0)) {
        finish(st, ST_NAN, 0);
        return;
    }
    st->k = 1;
    begin_iteration(st, tot[0]);                              // <r_hat_0, r> = <r, r>
}

__device__ inline void finish_gamma(SolverState* st, const double* tot, int step) {   // (7) / (14)
    st->gamma = tot[0];
    if (st->gamma == 0.0) {
        finish(st, ST_BREAKDOWN, step);
        return;
    }
    st->alpha = st->rho0 / st->gamma;
    if (step == 7) st->alpha1 = st->alpha;   // the alpha of step (10), applied in the last kernel
}

__device__ inline void finish_rho(SolverState* st, const double* tot) {               // (11)
    st->rho1 = tot[0];
    st->beta = st->alpha * st->rho1 / st->rho0;
    st->rho0 = st->rho1;
}

__device__ inline void finish_omega(SolverState* st, const double* tot) {             // (19)-(23)
    double omega_1 = tot[0], mu = tot[1], nu = tot[2], tau = tot[3], omega_2 = tot[4];
    if (mu == 0.) {
        finish(st, ST_BREAKDOWN, 20);
        return;
    }
    tau -= nu * nu / mu;                                      // (21)
    st->mu = mu;
    st->nu = nu;
    st->tau = tau;
    if (tau == 0.0) {
        finish(st, ST_TAU0, 21);
        return;
    }
    omega_2 = (omega_2 - (nu * omega_1) / mu) / tau;          // (22)
    omega_1 = (omega_1 - nu * omega_2) / mu;                  // (23)
    st->omega1 = omega_1;
    st->omega2 = omega_2;
}

__device__ inline void finish_update(SolverState* st, const double* tot) {            // (25) check, (3), (4)
    const double rnorm = sqrt(tot[0]);
    st->rnorm = rnorm;
    if (rnorm <= st->tol && st->k > 1) {
        finish(st, ST_CONVERGED, 0);
        return;
    }
    if (isnan(rnorm)) {
        finish(st, ST_NAN, 0);
        return;
    }
    st->k += 1;
    begin_iteration(st, tot[1]);
}

// ---------------------------------------------------------------------------
// operator rows: p[0..5] = W,E,S,N,B,T off-diagonals, p[6] = centre (general
// operator only); z[0..6] = C,W,E,S,N,B,T values of the SpMV operand
// ---------------------------------------------------------------------------
template <bool UNIT>
struct NCoef {
    static constexpr int value = UNIT ? 6 : 7;
};

template <typename T, bool UNIT>
__device__ __forceinline__ T apply_pre(const T* p, const T (&z)[7]) {
    T y = UNIT ? z[0] : p[6] * z[0];
    y += p[0] * z[1];
    y += p[1] * z[2];
    y += p[2] * z[3];
    y += p[3] * z[4];
    y += p[4] * z[5];
    y += p[5] * z[6];
    return y;
}

template <typename T, bool UNIT, int NP>
__host__ __device__ inline void set_coef_streams(const OpT<T>& op, const T* (&ps)[NP]) {
#pragma unroll
    for (int q = 0; q < 6; q++) ps[q] = op.off + q * op.n;
    if (!UNIT) ps[6] = op.c;
}

// ---------------------------------------------------------------------------
// fused stencil functors (plain data, built on the host)
//   zs[NZ] / zc(a, b):   the SpMV operand z = zc(zs[0][c], zs[1][c])
//   ps[NP]:              per-cell streams staged for the centre step
//   center(c, z, p, acc): writes, the SpMV row, dot-product terms
//   done(st, tot):       the scalar step, by the block finishing the last item
// ---------------------------------------------------------------------------

// K0: r = b - Op x; r_hat_0 = r; u = 0; sums <r,r>, <b,b>.  (The reference
// also zeroes v and w in step (1); every iteration writes both before it
// reads them -- v in step (6), w in step (13) -- so they are left alone.)
template <typename T, bool UNIT>
struct FInit {
    using type = T;
    static constexpr int Q = 2, NZ = 1, NC = NCoef<UNIT>::value, NP = NC + 1;
    static constexpr bool kCheckDone = false;
    static constexpr bool kPairs = false;   // two cells per thread (see launch_march)
    const T* zs[2];   // x
    const T* ps[NP];  // coefficients, b
    T *r, *rh, *u;
    __device__ void load(const SolverState*) {}
    __device__ T zc(T a, T) const { return a; }
    __device__ void center(int64_t c, const T (&zz)[7], const T* p, double* acc) const {
        const T bc = p[NC];
        const T rr = bc - apply_pre<T, UNIT>(p, zz);
        r[c] = rr;
        rh[c] = rr;
        u[c] = T(0);
        acc[0] += (double)rr * (double)rr;
        acc[1] += (double)bc * (double)bc;
    }
    __device__ void done(SolverState* st, const double* tot) const { finish_init(st, tot); }
};

// The four SpMV kernels store only their products v, s, w and t.  The vectors
// of the middle of an iteration -- u of step (5), r of (8), v of (12), r and s
// of (16)-(17) -- are operands formed while staging, and a later kernel that
// needs one again forms it again from the r, u, v, s and w it comes from, with
// the same expression (so the same bits): none of those five is overwritten
// before the last kernel.  That takes five stores and one load of n values
// out of an iteration (464 -> 416 bytes per cell in FP64): the 256^3 TVD step
// went from 12.05 to 11.33 ms, the 384^3 FP32-refine step from 24.4 to 22.7.

// K1: (5) u = r - beta u; (6) v = Op u; (7) gamma = <v, r_hat_0>
template <typename T, bool UNIT>
struct FStep1 {
    using type = T;
    static constexpr int Q = 1, NZ = 2, NC = NCoef<UNIT>::value, NP = NC + 1;
    static constexpr bool kCheckDone = true;
    static constexpr bool kPairs = sizeof(T) == 4;   // two cells per thread (see launch_march)
    const T* zs[2];   // r, u
    const T* ps[NP];  // coefficients, r_hat_0
    T* v;
    T beta;
    __device__ void load(const SolverState* st) { beta = (T)st->beta; }
    __device__ T zc(T r, T u) const { return r - beta * u; }
    __device__ void center(int64_t c, const T (&zz)[7], const T* p, double* acc) const {
        const T vc = apply_pre<T, UNIT>(p, zz);
        v[c] = vc;
        acc[0] += (double)vc * (double)p[NC];
    }
    __device__ void done(SolverState* st, const double* tot) const { finish_gamma(st, tot, 7); }
};

// K2: (8) r = r - alpha v; (9) s = Op r; (11) rho1 = <r_hat_0, s>.  Step
// (10), x = x + alpha u, waits for K5 (x is read by nothing in between),
// which saves x's read and write here.
template <typename T, bool UNIT>
struct FStep2 {
    using type = T;
    static constexpr int Q = 1, NZ = 2, NC = NCoef<UNIT>::value, NP = NC + 1;
    static constexpr bool kCheckDone = true;
    static constexpr bool kPairs = sizeof(T) == 4;   // two cells per thread (see launch_march)
    const T* zs[2];   // v, r
    const T* ps[NP];  // coefficients, r_hat_0
    T* s;
    T alpha;
    __device__ void load(const SolverState* st) { alpha = (T)st->alpha; }
    __device__ T zc(T v, T r) const { return -alpha * v + r; }
    __device__ void center(int64_t c, const T (&zz)[7], const T* p, double* acc) const {
        const T sc = apply_pre<T, UNIT>(p, zz);
        s[c] = sc;
        acc[0] += (double)p[NC] * (double)sc;
    }
    __device__ void done(SolverState* st, const double* tot) const { finish_rho(st, tot); }
};

// K3: (12) v = s - beta v; (13) w = Op v; (14) gamma = <w, r_hat_0>
template <typename T, bool UNIT>
struct FStep3 {
    using type = T;
    static constexpr int Q = 1, NZ = 2, NC = NCoef<UNIT>::value, NP = NC + 1;
    static constexpr bool kCheckDone = true;
    static constexpr bool kPairs = sizeof(T) == 4;   // two cells per thread (see launch_march)
    const T* zs[2];   // s, v
    const T* ps[NP];  // coefficients, r_hat_0
    T* w;
    T beta;
    __device__ void load(const SolverState* st) { beta = (T)st->beta; }
    __device__ T zc(T s, T v) const { return s - beta * v; }
    __device__ void center(int64_t c, const T (&zz)[7], const T* p, double* acc) const {
        const T wc = apply_pre<T, UNIT>(p, zz);
        w[c] = wc;
        acc[0] += (double)wc * (double)p[NC];
    }
    __device__ void done(SolverState* st, const double* tot) const { finish_gamma(st, tot, 14); }
};

// r after steps (8) and (16), from the iterate's r, the v of step (6) and the
// s of step (9): v' = s - beta v (12), r' = r - alpha1 v (8), r'' = r' - alpha v'
template <typename T>
__device__ __forceinline__ T r_of_16(T r, T v, T s, T alpha1, T alpha, T beta) {
    const T v12 = s - beta * v;
    const T r8 = -alpha1 * v + r;
    return -alpha * v12 + r8;
}

// K4: (16) r = r - alpha v; (17) s = s - alpha w; (18) t = Op s;
//     (19)-(20) <r,s>, <s,s>, <s,t>, <t,t>, <r,t>; (21)-(23).  Step (16)'s
//     terms come from the r, v and s staged here (kRaw: center3 also gets the
//     second staged operand's own value, the s of step (9)).
template <typename T, bool UNIT>
struct FStep4 {
    using type = T;
    static constexpr int Q = 5, NZ = 2, NC = NCoef<UNIT>::value, NP = NC + 2;
    static constexpr bool kCheckDone = true;
    static constexpr bool kPairs = sizeof(T) == 4;   // two cells per thread (see launch_march)
    static constexpr bool kRaw = true;
    const T* zs[2];   // w, s
    const T* ps[NP];  // coefficients, r, v
    T* t;
    T alpha, alpha1, beta;
    __device__ void load(const SolverState* st) {
        alpha = (T)st->alpha;
        alpha1 = (T)st->alpha1;
        beta = (T)st->beta;
    }
    __device__ T zc(T w, T s) const { return -alpha * w + s; }
    __device__ void center3(int64_t c, const T (&zz)[7], T s9, const T* p, double* acc) const {
        const T rn = r_of_16(p[NC], p[NC + 1], s9, alpha1, alpha, beta);
        const T tc = apply_pre<T, UNIT>(p, zz);
        t[c] = tc;
        const double dr = rn, ds = zz[0], dt = tc;
        acc[0] += dr * ds;
        acc[1] += ds * ds;
        acc[2] += ds * dt;
        acc[3] += dt * dt;
        acc[4] += dr * dt;
    }
    __device__ void done(SolverState* st, const double* tot) const { finish_omega(st, tot); }
};

// ||b - A x||_2 with the general operator, written to *out
template <typename T>
struct FResidual {
    using type = T;
    static constexpr int Q = 1, NZ = 1, NP = 8;
    static constexpr bool kCheckDone = false;
    static constexpr bool kPairs = false;   // two cells per thread (see launch_march)
    const T* zs[2];   // x
    const T* ps[NP];  // 7 coefficients, b
    double* out;
    __device__ void load(const SolverState*) {}
    __device__ T zc(T a, T) const { return a; }
    __device__ void center(int64_t, const T (&zz)[7], const T* p, double* acc) const {
        const double r = (double)p[7] - (double)apply_pre<T, false>(p, zz);
        acc[0] += r * r;
    }
    __device__ void done(SolverState*, const double* tot) const { *out = sqrt(tot[0]); }
};

// Ahat[q][c] = A[q][c] * invd[neighbour_q(c)] (removed neighbours read 0)
struct FFold {
    using type = double;
    static constexpr int Q = 0, NZ = 1, NP = 6;
    static constexpr bool kCheckDone = false;
    static constexpr bool kPairs = false;   // two cells per thread (see launch_march)
    const double* zs[2];   // invd
    const double* ps[NP];  // the 6 off-diagonals of A
    double* ahat;
    int64_t n;
    __device__ void load(const SolverState*) {}
    __device__ double zc(double a, double) const { return a; }
    __device__ void center(int64_t c, const double (&zz)[7], const double* p, double*) const {
#pragma unroll
        for (int q = 0; q < 6; q++) ahat[q * n + c] = p[q] * zz[q + 1];
    }
    __device__ void done(SolverState*, const double*) const {}
};

// The same, rounded to FP32: the operator of the FP32 inner solves, written
// without an FP64 copy
struct FFold32 {
    using type = double;
    static constexpr int Q = 0, NZ = 1, NP = 6;
    static constexpr bool kCheckDone = false;
    static constexpr bool kPairs = false;   // two cells per thread (see launch_march)
    const double* zs[2];   // invd
    const double* ps[NP];  // the 6 off-diagonals of A
    float* ahat;
    int64_t n;
    __device__ void load(const SolverState*) {}
    __device__ double zc(double a, double) const { return a; }
    __device__ void center(int64_t c, const double (&zz)[7], const double* p, double*) const {
#pragma unroll
        for (int q = 0; q < 6; q++) ahat[q * n + c] = (float)(p[q] * zz[q + 1]);
    }
    __device__ void done(SolverState*, const double*) const {}
};

// K0 with the Jacobi fold, one pass instead of FFold then FInit: Ahat[q][c] =
// A[q][c] * invd[neighbour_q(c)] written, then r = b - Ahat y from those
// values, r_hat_0 = r, u = 0; sums <r,r>, <b,b>.  The products and sums are
// the two kernels' own, in their order, so the results are the same bits.
// Split operands (kSplit): the kernel hands over both staged arrays' seven
// values, invd and y, instead of one combined operand.
struct FFoldInit {
    using type = double;
    static constexpr int Q = 2, NZ = 2, NP = 7;
    static constexpr bool kCheckDone = false;
    static constexpr bool kPairs = false;
    static constexpr bool kSplit = true;
    const double* zs[2];   // invd, y
    const double* ps[NP];  // the 6 off-diagonals of A, b
    double *ahat, *r, *rh, *u;
    int64_t n;
    __device__ void load(const SolverState*) {}
    __device__ double zc(double a, double) const { return a; }   // (the combined operand is not used)
    __device__ void center2(int64_t c, const double (&iv)[7], const double (&y)[7], const double* p,
                            double* acc) const {
        double a[6];
#pragma unroll
        for (int q = 0; q < 6; q++) {
            a[q] = p[q] * iv[q + 1];
            ahat[q * n + c] = a[q];
        }
        double yy = y[0];   // apply_pre<double, true>(a, y)
        yy += a[0] * y[1];
        yy += a[1] * y[2];
        yy += a[2] * y[3];
        yy += a[3] * y[4];
        yy += a[4] * y[5];
        yy += a[5] * y[6];
        const double bc = p[6];
        const double rr = bc - yy;
        r[c] = rr;
        rh[c] = rr;
        u[c] = 0.;
        acc[0] += rr * rr;
        acc[1] += bc * bc;
    }
    __device__ void done(SolverState* st, const double* tot) const { finish_init(st, tot); }
};

template <class K, class = void>
struct SplitOperands {
    static constexpr bool value = false;
};
template <class K>
struct SplitOperands<K, std::void_t<decltype(K::kSplit)>> {
    static constexpr bool value = K::kSplit;
};

// functors whose center step also takes the second staged operand's own value
template <class K, class = void>
struct RawOperand {
    static constexpr bool value = false;
};
template <class K>
struct RawOperand<K, std::void_t<decltype(K::kRaw)>> {
    static constexpr bool value = K::kRaw;
};

// ---------------------------------------------------------------------------
// the functors of the init kernel and of one iteration over the vectors vs,
// shared by the single-grid and the slab drivers
// ---------------------------------------------------------------------------
template <typename T, bool UNIT>
FInit<T, UNIT> make_init(const OpT<T>& op, const VecsT<T>& vs) {
    using F = FInit<T, UNIT>;
    F f{};
    f.zs[0] = vs.x;
    set_coef_streams<T, UNIT, F::NP>(op, f.ps);
    f.ps[F::NC] = vs.b;
    f.r = vs.r;
    f.rh = vs.rh;
    f.u = vs.u;
    return f;
}
template <typename T, bool UNIT>
FStep1<T, UNIT> make_step1(const OpT<T>& op, const VecsT<T>& vs) {
    FStep1<T, UNIT> f{};
    f.zs[0] = vs.r;
    f.zs[1] = vs.u;
    set_coef_streams<T, UNIT, FStep1<T, UNIT>::NP>(op, f.ps);
    f.ps[NCoef<UNIT>::value] = vs.rh;
    f.v = vs.v;
    return f;
}
template <typename T, bool UNIT>
FStep2<T, UNIT> make_step2(const OpT<T>& op, const VecsT<T>& vs) {
    constexpr int NC = NCoef<UNIT>::value;
    FStep2<T, UNIT> f{};
    f.zs[0] = vs.v;
    f.zs[1] = vs.r;
    set_coef_streams<T, UNIT, FStep2<T, UNIT>::NP>(op, f.ps);
    f.ps[NC] = vs.rh;
    f.s = vs.s;
    return f;
}
template <typename T, bool UNIT>
FStep3<T, UNIT> make_step3(const OpT<T>& op, const VecsT<T>& vs) {
    FStep3<T, UNIT> f{};
    f.zs[0] = vs.s;
    f.zs[1] = vs.v;
    set_coef_streams<T, UNIT, FStep3<T, UNIT>::NP>(op, f.ps);
    f.ps[NCoef<UNIT>::value] = vs.rh;
    f.w = vs.w;
    return f;
}
template <typename T, bool UNIT>
FStep4<T, UNIT> make_step4(const OpT<T>& op, const VecsT<T>& vs) {
    constexpr int NC = NCoef<UNIT>::value;
    FStep4<T, UNIT> f{};
    f.zs[0] = vs.w;
    f.zs[1] = vs.s;
    set_coef_streams<T, UNIT, FStep4<T, UNIT>::NP>(op, f.ps);
    f.ps[NC] = vs.r;
    f.ps[NC + 1] = vs.v;
    f.t = vs.t;
    return f;
}
inline FResidual<double> make_residual(const OpT<double>& op, const double* x, const double* b, double* out) {
    FResidual<double> f{};
    f.zs[0] = x;
    set_coef_streams<double, false, 8>(op, f.ps);
    f.ps[7] = b;
    f.out = out;
    return f;
}
inline FFold make_fold(const double* diag, const double* invd, double* ahat, int64_t n) {
    FFold f{};
    f.zs[0] = invd;
    for (int q = 0; q < 6; q++) f.ps[q] = diag + (q + 1) * n;
    f.ahat = ahat;
    f.n = n;
    return f;
}

// ---------------------------------------------------------------------------
// item reduction: partials are indexed by item; the item whose counter
// increment completes the set sums them in item order.
// ---------------------------------------------------------------------------
template <int Q>
__device__ bool item_reduce(double (&v)[Q], double* __restrict__ partials, int item, int nitems,
                            unsigned int* counter, double (&tot)[Q]) {
    __shared__ double sh[32 * kMaxQ];
    __shared__ bool is_last;
    block_sum<Q>(v, sh);
    const int tid = thread_linear();
    if (tid == 0) {
#pragma unroll
        for (int q = 0; q < Q; q++) partials[q * kMaxBlocks + item] = v[q];
        __threadfence();
        const unsigned prev = atomicAdd(counter, 1u);
        is_last = (prev == (unsigned)nitems - 1);
    }
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    double a[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) a[q] = 0.;
    const int nt = blockDim.x * blockDim.y;
    for (int b = tid; b < nitems; b += nt) {
#pragma unroll
        for (int q = 0; q < Q; q++) a[q] += __ldcg(partials + q * kMaxBlocks + b);
    }
    block_sum<Q>(a, sh);
#pragma unroll
    for (int q = 0; q < Q; q++) tot[q] = a[q];
    if (tid == 0) *counter = 0u;
    return true;
}

// ---------------------------------------------------------------------------
// asynchronous global -> shared copies (zero-filled when src_bytes == 0)
// ---------------------------------------------------------------------------
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int src = valid ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(src)
                 : "memory");
}
// The 16-byte copies of the operator's off-diagonals: their kernel reads them
// once and the next one only after all the others, so they are the first to leave
// L2 and the vectors that one kernel wrote are still there for the next (FP64
// 128^3 time step 1.76 -> 1.68 ms; no difference at 192^3 and 256^3, where the
// vectors alone are larger than L2).  L1: FP64 copies go through L1 (past it
// 256^3 took 12.6 ms for 12.1), the FP32 ones past it (256^3 refined solve
// 6.35 -> 6.23 ms; with every copy past it 1 % slower again).
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
    return p;
}
template <bool L1>
__device__ __forceinline__ void cp_async16_once(void* smem, const void* gmem, bool valid, uint64_t policy) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int src = valid ? 16 : 0;
    if constexpr (L1)
        asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(s), "l"(gmem), "r"(src),
                     "l"(policy)
                     : "memory");
    else
        asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(s), "l"(gmem), "r"(src),
                     "l"(policy)
                     : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Shared-memory elements of one stage of a marching block for functor K: a
// tile of tw x tj cells (tw = threads in x times cells per thread), operand
// rows padded by ic columns on each side (the halo column sits at ic - 1 and
// ic + tw), plus the per-cell streams.
template <class K>
__host__ __device__ constexpr size_t march_stage_elems(int tw, int tj, int ic) {
    return (size_t)K::NZ * (tw + 2 * ic) * (tj + 2) + (size_t)K::NP * tw * tj;
}
// Stages of the ring of planes.  While plane i is computed from planes i and
// i + 1, the stages up to i + depth - 1 are on their way: with two blocks a SM a
// kernel of the FP64 iteration has about 74 KB a SM in flight with four stages
// (256^3: steps at 5.7 TB/s with three; time step 12.08 -> 11.83 ms with four;
// five leave one block a SM, 15.2 ms).  The FP32 kernels run three blocks a SM
// with three stages (four stages, two blocks: 0.5 to 1 % slower).
template <typename T>
struct MarchDepth {
    static constexpr int value = sizeof(T) == 8 ? 4 : 3;
};
template <class K>
inline size_t march_smem_bytes(const MarchCfg& m) {
    const int ic = m.cpt;   // first interior column: one row segment of padding
    return MarchDepth<typename K::type>::value * march_stage_elems<K>(m.block.x * m.cpt, m.block.y, ic) *
           sizeof(typename K::type);
}

// two consecutive elements of shared memory in one load (16-byte aligned for
// double, 8-byte for float)
template <typename T>
struct Pair {
    T x, y;
};
template <typename T>
__device__ __forceinline__ Pair<T> ld_pair(const T* p) {
    if constexpr (sizeof(T) == 8) {
        const double2 v = *reinterpret_cast<const double2*>(p);
        return Pair<T>{(T)v.x, (T)v.y};
    } else {
        const float2 v = *reinterpret_cast<const float2*>(p);
        return Pair<T>{(T)v.x, (T)v.y};
    }
}

// ---------------------------------------------------------------------------
// the persistent plane-marching kernel.  CPT cells per thread along k: with
// CPT = 2 (even n2) every staged row segment of a thread is one 16-byte copy
// (8 bytes for FP32), halving the per-cell copies, index arithmetic and
// barrier waits; the operand rows are padded so those copies stay aligned.
// ---------------------------------------------------------------------------
// Register budgets, measured at 256^3: two cells per thread held to 80
// registers (steps 1 and 3: 0.264 -> 0.257 ms); one cell per thread up to 128,
// two blocks per SM (held to 80 registers, steps 2 and 4 went from
// 0.343 / 0.353 ms to 0.408 / 0.433 ms, also when the maximum shared-memory
// carveout then let three blocks in; that carveout also slowed steps 1 and 3
// to 0.354 ms, so the default carveout stays).
// HALO (slabs): the planes before the first and after the last plane of the
// grid come from m.halo when set.
// Blocks per SM the register budget is set for: three (80 registers) with
// two cells per thread, two (128) with one.  Step 4 (two staged operands,
// eight streams, five FP64 dot products) takes two blocks of 128 registers
// with two cells per thread too: held to 80, the FP32 step 4 of the
// refinement ran 1.66 ms at 512^3 (64 % of copy bandwidth), with 128
// registers 1.18 ms (90 %).
template <class K, int CPT>
struct MarchMinBlocks {
    static constexpr int value = CPT == 2 ? 3 : 2;
};
template <typename T, bool UNIT, int CPT>
struct MarchMinBlocks<FStep4<T, UNIT>, CPT> {
    static constexpr int value = 2;
};

template <class K, int CPT = 1, bool HALO = false, bool PAIR = false>
__global__ void __launch_bounds__(256, MarchMinBlocks<K, CPT>::value) k_march(GridDev g, K kern, SolverState* st, double* partials,
                                                                   MarchCfg m) {
    using T = typename K::type;
    constexpr int NZ = K::NZ, NP = K::NP;
    constexpr int QA = K::Q > 0 ? K::Q : 1;
    constexpr int VEC = 16 / (int)sizeof(T);    // cells of one 16-byte copy
    static_assert(!PAIR || VEC % CPT == 0, "16-byte staging: a copy covers whole thread segments");
    constexpr int IC = PAIR ? VEC : CPT;        // first interior column of a staged operand row
    constexpr int CB = CPT * (int)sizeof(T);    // bytes of one thread's row segment
    constexpr int D = MarchDepth<T>::value;
    const uint64_t once = evict_first_policy();
    pdl_wait();
    pdl_launch();
    if (K::kCheckDone && st->done) return;
    K k = kern;
    k.load(st);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(smem_raw);
    __shared__ int s_item;
    const int TK = blockDim.x, TJ = blockDim.y;
    const int TW = TK * CPT;                    // tile width in cells
    const int W = TW + 2 * IC, H = TJ + 2;
    const int ZT = W * H;                       // one staged operand tile
    const int NCT = TW * TJ;                    // cells of the tile
    const int STAGE = NZ * ZT + NP * NCT;       // elements per stage
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = tx + TK * ty;
    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
    const int n0c = n0 / g.ncomp;               // planes of one field component
    const int p0 = g.periodic[0], p1 = g.periodic[1], p2 = g.periodic[2];
    const int64_t plane = (int64_t)n1 * n2;
    const int tiles = m.tiles_x * m.tiles_y;

    // Geometry of one work item for this thread.
    struct Geo {
        int i0, i1;
        int cb;        // first stacked plane of this item's component
        bool inside, hS, hN, hB, hT;
        int64_t o_c, o_s, o_n, o_b, o_t, o_own;
        int64_t o_pair;   // PAIR: in-plane offset of this thread's pair of stream cells (-1: outside)
        int64_t o_op;     // PAIR: in-plane offset of this thread's operand copy (-1: zero)
    };
    // PAIR: every value staged as part of a 16-byte copy of VEC cells (FP64
    // with one cell per thread, FP32 with two: row length and tile width
    // multiples of VEC).  The per-cell streams: the first half of the threads
    // copies the even-numbered streams and the second half the odd ones, one
    // 16-byte copy each -- half the copies and address arithmetic of one
    // copy per thread and stream (256^3 FP64 step 4: 0.316 -> 0.298 ms).
    static_assert(!PAIR || VEC / CPT == 2, "16-byte staging: two thread sets");
    const int npairs = NCT / VEC;               // 16-byte copies per stream and plane (half the threads)
    const int par = tid >= npairs;
    const int e_pair = tid - par * npairs;
    const int hw = TW / VEC > 0 ? TW / VEC : 1;   // copies per row (PAIR needs TW % VEC == 0)
    const int pr_row = e_pair / hw, pr_col = VEC * (e_pair - pr_row * hw);
    // PAIR: the operand tiles' rows 0 .. TJ+1 (j0-1 .. j0+TJ) as 16-byte copies,
    // then the single halo cells k0-1 and k0+TW of rows 1 .. TJ; thread tid
    // makes one copy of every operand array (op_kind 2: 16 bytes, 1: one
    // cell, 0: none) -- (TJ+2) TW/VEC + 2 TJ copies, all threads alike, in place
    // of one copy per cell plus the halo copies of the edge threads (256^3
    // FP64 step 4: 0.298 -> 0.285 ms, 6.1 TB/s; the FP32 kernels on 64 x 8
    // tiles run two cells per thread this way, 512^3 FP32-refine solve 52.8
    // -> 51.7 ms)
    int op_kind = 0, op_row = 0, op_col = 0, op_dk = 0;
    if constexpr (PAIR) {
        const int npr = (TJ + 2) * hw;
        if (tid < npr) {
            op_kind = 2;
            op_row = tid / hw;
            op_dk = VEC * (tid - op_row * hw);
            op_col = IC + op_dk;
        } else if (tid < npr + 2 * TJ) {
            const int e = tid - npr;
            op_kind = 1;
            op_row = 1 + (e >> 1);
            op_dk = (e & 1) ? TW : -1;
            op_col = IC + op_dk;
        }
    }
    // in-plane position (j, kx) -> wrapped offset, or -1 when outside (zero)
    auto jk_offset = [&](int j, int kx) -> int64_t {
        if (j < 0) {
            if (!p1) return -1;
            j += n1;
        } else if (j >= n1) {
            if (!p1) return -1;
            j -= n1;
        }
        if (kx < 0) {
            if (!p2) return -1;
            kx += n2;
        } else if (kx >= n2) {
            if (!p2) return -1;
            kx -= n2;
        }
        if ((unsigned)j >= (unsigned)n1 || (unsigned)kx >= (unsigned)n2) return -1;
        return (int64_t)j * n2 + kx;
    };
    auto geometry = [&](int item) {
        Geo G;
        const int tile_id = item % tiles;
        const int chunk = item / tiles;
        const int kk = (tile_id % m.tiles_x) * TW + CPT * tx;   // this thread's first cell
        const int jj = (tile_id / m.tiles_x) * TJ + ty;
        // runs of planes never cross from one field component to the next
        const int comp = g.ncomp > 1 ? chunk / m.cpc : 0;
        G.cb = comp * n0c;
        G.i0 = G.cb + (chunk - comp * m.cpc) * m.planes;
        G.i1 = min(G.i0 + m.planes, G.cb + n0c);
        // (n2 is even when CPT = 2, so a thread's cells are both inside or both outside)
        G.inside = jj < n1 && kk < n2;
        const bool edge = jj <= n1 && kk <= n2;   // the first row / column past the grid is read as halo
        G.hS = G.inside && ty == 0;
        G.hN = G.inside && ty == TJ - 1;
        G.hB = G.inside && tx == 0;
        G.hT = G.inside && tx == TK - 1;
        G.o_c = edge ? jk_offset(jj, kk) : -1;
        G.o_s = G.hS ? jk_offset(jj - 1, kk) : -1;
        G.o_n = G.hN ? jk_offset(jj + 1, kk) : -1;
        G.o_b = G.hB ? jk_offset(jj, kk - 1) : -1;
        G.o_t = G.hT ? jk_offset(jj, kk + CPT) : -1;
        G.o_own = G.inside ? (int64_t)jj * n2 + kk : 0;
        G.o_pair = G.o_op = -1;
        if constexpr (PAIR) {
            const int tj0 = (tile_id / m.tiles_x) * TJ, tk0 = (tile_id % m.tiles_x) * TW;
            const int pj = tj0 + pr_row, pk = tk0 + pr_col;
            G.o_pair = (pj < n1 && pk < n2) ? (int64_t)pj * n2 + pk : -1;
            // a pair past n2 starts at the wrapped (or removed) first cell; its
            // second cell is never read
            if (op_kind) G.o_op = jk_offset(tj0 - 1 + op_row, tk0 + op_dk);
        }
        return G;
    };
    auto slot_of = [&](const Geo& G, int p) { return (p - G.i0 + 1) % D; };
    // Stage plane p into its ring slot: operand inputs with halo, and (when
    // `full`) the per-cell streams.  Out-of-range planes are zeros.
    auto stage = [&](const Geo& G, int p, bool full) {
        T* sb = smem + (size_t)slot_of(G, p) * STAGE;
        bool pv = true;
        int pp = p - G.cb;   // plane within the component, wrapped on a periodic x
        if (pp < 0) {
            pv = p0;
            pp += n0c;
        } else if (pp >= n0c) {
            pv = p0;
            pp -= n0c;
        }
        const int64_t base = (int64_t)(G.cb + pp) * plane;
        const int col = IC + CPT * tx;
#pragma unroll
        for (int z = 0; z < NZ; z++) {
            const T* src = k.zs[z];
            T* zt = sb + z * ZT;
            int64_t zb = base;
            bool zv = pv;
            if constexpr (HALO) {
                const int hside = p - G.cb < 0 ? 0 : (p - G.cb >= n0c ? 1 : -1);   // a plane past the slab
                const void* nb = hside == 0 ? m.halo[z][0] : (hside == 1 ? m.halo[z][1] : nullptr);
                if (nb) {   // the neighbour's plane, exchanged into a local buffer
                    src = static_cast<const T*>(nb) + (int64_t)(G.cb / n0c) * plane;   // [component][plane]
                    zb = 0;
                    zv = true;
                }
            }
            if constexpr (PAIR) {
                if (op_kind == 2)
                    cp_async<16>(zt + op_row * W + op_col, src + zb + (G.o_op < 0 ? 0 : G.o_op), zv && G.o_op >= 0);
                else if (op_kind == 1)
                    cp_async<(int)sizeof(T)>(zt + op_row * W + op_col, src + zb + (G.o_op < 0 ? 0 : G.o_op),
                                             zv && G.o_op >= 0);
                continue;
            }
            cp_async<CB>(zt + (ty + 1) * W + col, src + zb + (G.o_c < 0 ? 0 : G.o_c), zv && G.o_c >= 0);
            if (G.hS) cp_async<CB>(zt + col, src + zb + (G.o_s < 0 ? 0 : G.o_s), zv && G.o_s >= 0);
            if (G.hN)
                cp_async<CB>(zt + (TJ + 1) * W + col, src + zb + (G.o_n < 0 ? 0 : G.o_n), zv && G.o_n >= 0);
            if (G.hB)
                cp_async<sizeof(T)>(zt + (ty + 1) * W + IC - 1, src + zb + (G.o_b < 0 ? 0 : G.o_b),
                                    zv && G.o_b >= 0);
            if (G.hT)
                cp_async<sizeof(T)>(zt + (ty + 1) * W + IC + TW, src + zb + (G.o_t < 0 ? 0 : G.o_t),
                                    zv && G.o_t >= 0);
        }
        if constexpr (PAIR) {
            if (full) {
                T* pt = sb + NZ * ZT + pr_row * TW + pr_col;
#pragma unroll
                for (int q = 0; q < NP; q++)
                    if ((q & 1) == par) {
                        const T* src = k.ps[q] + base + (G.o_pair < 0 ? 0 : G.o_pair);
                        if (q < 6)   // off-diagonals
                            cp_async16_once<sizeof(T) == 8>(pt + q * NCT, src, G.o_pair >= 0, once);
                        else
                            cp_async<16>(pt + q * NCT, src, G.o_pair >= 0);
                    }
            }
            return;
        }
        if (full && G.inside) {
            T* pt = sb + NZ * ZT + ty * TW + CPT * tx;
#pragma unroll
            for (int q = 0; q < NP; q++) cp_async<CB>(pt + q * NCT, k.ps[q] + base + G.o_own, true);
        }
    };
    // prologue of an item: planes i0-1 (operand only), i0 .. i0+D-2
    auto prologue = [&](const Geo& G) {
        stage(G, G.i0 - 1, false);
        cp_async_commit();
        stage(G, G.i0, true);
        cp_async_commit();
#pragma unroll
        for (int d = 1; d < D - 1; d++) {
            if (G.i0 + d <= G.i1) stage(G, G.i0 + d, G.i0 + d < G.i1);
            cp_async_commit();
        }
    };
    auto zval = [&](const T* sb, int row, int col) -> T {
        const T a = sb[row * W + col];
        const T b = NZ > 1 ? sb[ZT + row * W + col] : T(0);
        return k.zc(a, b);
    };

    // Items come from the queue one ahead: the next index is fetched when an
    // item starts, and the next item's prologue copies are issued before the
    // current item's reduction, so the queue atomic, the reduction and the
    // first planes' DRAM latency overlap.
    __shared__ int s_next;
    if (tid == 0) s_item = (int)atomicAdd(&st->queue, 1u);
    __syncthreads();
    int item = s_item;
    Geo G = geometry(item < m.nitems ? item : 0);
    if (item < m.nitems) prologue(G);
    while (item < m.nitems) {
        if (tid == 0) s_next = (int)atomicAdd(&st->queue, 1u);
        double acc[QA];
#pragma unroll
        for (int q = 0; q < QA; q++) acc[q] = 0.;
        cp_async_wait<D - 2>();                 // planes i0-1 and i0
        __syncthreads();
        constexpr bool SPLIT = SplitOperands<K>::value;
        // the thread's operand values of planes i - 1 and i (split operands: of
        // both arrays), kept from the plane before: L1 and shared memory run at
        // 70 % of their rate, and reading plane i's again cost 1.3 % at 256^3
        T zprev[CPT], zthis[CPT];
        T zprev_b = T(0), zthis_b = T(0);
        const T* sp = smem + (size_t)slot_of(G, G.i0 - 1) * STAGE;
        const T* s0 = smem + (size_t)slot_of(G, G.i0) * STAGE;
        if constexpr (SPLIT) {
            const int at = (ty + 1) * W + IC + tx;
            zprev[0] = G.inside ? sp[at] : T(0);
            zprev_b = G.inside ? sp[ZT + at] : T(0);
            zthis[0] = G.inside ? s0[at] : T(0);
            zthis_b = G.inside ? s0[ZT + at] : T(0);
        } else {
#pragma unroll
            for (int c = 0; c < CPT; c++) {
                zprev[c] = G.inside ? zval(sp, ty + 1, IC + CPT * tx + c) : T(0);
                zthis[c] = G.inside ? zval(s0, ty + 1, IC + CPT * tx + c) : T(0);
            }
        }
        for (int i = G.i0; i < G.i1; i++) {
            if constexpr (D > 3) cp_async_wait<D - 3>();   // planes i and i+1 have landed
            __syncthreads();                    // and every thread is done with plane i-1
            if (i + D - 1 <= G.i1) stage(G, i + D - 1, i + D - 1 < G.i1);   // in the slot of plane i-1
            cp_async_commit();
            if constexpr (D == 3) {             // plane i+1 has too
                cp_async_wait<1>();
                __syncthreads();
            }
            const T* sb = smem + (size_t)slot_of(G, i) * STAGE;
            const T* sn = smem + (size_t)slot_of(G, i + 1) * STAGE;
            if (G.inside) {
                if constexpr (SPLIT) {
                    static_assert(CPT == 1, "split operands run one cell per thread");
                    const int col = IC + tx;
                    auto raw = [&](const T* b, int z, int row, int cc) { return b[z * ZT + row * W + cc]; };
                    const T a0 = zthis[0], b0 = zthis_b;
                    const T an = raw(sn, 0, ty + 1, col), bn = raw(sn, 1, ty + 1, col);
                    const T za[7] = {a0, zprev[0], an, raw(sb, 0, ty, col), raw(sb, 0, ty + 2, col),
                                     raw(sb, 0, ty + 1, col - 1), raw(sb, 0, ty + 1, col + 1)};
                    const T zb[7] = {b0, zprev_b, bn, raw(sb, 1, ty, col), raw(sb, 1, ty + 2, col),
                                     raw(sb, 1, ty + 1, col - 1), raw(sb, 1, ty + 1, col + 1)};
                    T pv[NP];
#pragma unroll
                    for (int q = 0; q < NP; q++) pv[q] = sb[NZ * ZT + q * NCT + tid];
                    k.center2((int64_t)i * plane + G.o_own, za, zb, pv, acc);
                    zprev[0] = a0;
                    zprev_b = b0;
                    zthis[0] = an;
                    zthis_b = bn;
                } else if constexpr (CPT == 1) {
                    const int col = IC + tx;
                    const T zcur = zthis[0], znext = zval(sn, ty + 1, col);
                    const T z7[7] = {zcur, zprev[0], znext, zval(sb, ty, col), zval(sb, ty + 2, col),
                                     zval(sb, ty + 1, col - 1), zval(sb, ty + 1, col + 1)};
                    T pv[NP];
#pragma unroll
                    for (int q = 0; q < NP; q++) pv[q] = sb[NZ * ZT + q * NCT + tid];
                    if constexpr (RawOperand<K>::value)
                        k.center3((int64_t)i * plane + G.o_own, z7, sb[ZT + (ty + 1) * W + col], pv, acc);
                    else
                        k.center((int64_t)i * plane + G.o_own, z7, pv, acc);
                    zprev[0] = zcur;
                    zthis[0] = znext;
                } else if constexpr (CPT == 2) {
                    // the thread's two cells as one 16-byte (8-byte for FP32)
                    // shared-memory load per row: consecutive threads read
                    // consecutive pairs, without bank conflicts
                    const int col = IC + 2 * tx;
                    auto zpair = [&](const T* b, int row, T& z0, T& z1) {
                        const Pair<T> a = ld_pair(b + row * W + col);
                        Pair<T> c2{T(0), T(0)};
                        if constexpr (NZ > 1) c2 = ld_pair(b + ZT + row * W + col);
                        z0 = k.zc(a.x, c2.x);
                        z1 = k.zc(a.y, c2.y);
                    };
                    const T zc0 = zthis[0], zc1 = zthis[1];
                    T zn0, zn1, zs0, zs1, zt0, zt1;
                    zpair(sn, ty + 1, zn0, zn1);
                    zpair(sb, ty, zs0, zs1);
                    zpair(sb, ty + 2, zt0, zt1);
                    const T zw = zval(sb, ty + 1, col - 1), ze = zval(sb, ty + 1, col + 2);
                    T pv0[NP], pv1[NP];
#pragma unroll
                    for (int q = 0; q < NP; q++) {
                        const Pair<T> pq = ld_pair(sb + NZ * ZT + q * NCT + ty * TW + 2 * tx);
                        pv0[q] = pq.x;
                        pv1[q] = pq.y;
                    }
                    const T z70[7] = {zc0, zprev[0], zn0, zs0, zt0, zw, zc1};
                    const T z71[7] = {zc1, zprev[1], zn1, zs1, zt1, zc0, ze};
                    if constexpr (RawOperand<K>::value) {
                        const Pair<T> raw = ld_pair(sb + ZT + (ty + 1) * W + col);
                        k.center3((int64_t)i * plane + G.o_own, z70, raw.x, pv0, acc);
                        k.center3((int64_t)i * plane + G.o_own + 1, z71, raw.y, pv1, acc);
                    } else {
                        k.center((int64_t)i * plane + G.o_own, z70, pv0, acc);
                        k.center((int64_t)i * plane + G.o_own + 1, z71, pv1, acc);
                    }
                    zprev[0] = zc0;
                    zprev[1] = zc1;
                    zthis[0] = zn0;
                    zthis[1] = zn1;
                } else {
                    // four FP32 cells per thread: every row segment one 16-byte
                    // copy and one 16-byte shared-memory load
                    static_assert(CPT == 4 && sizeof(T) == 4, "four cells per thread: FP32");
                    const int col = IC + 4 * tx;
                    auto zquad = [&](const T* b, int row, T (&z)[4]) {
                        const float4 a = *reinterpret_cast<const float4*>(b + row * W + col);
                        float4 c2 = make_float4(0.f, 0.f, 0.f, 0.f);
                        if constexpr (NZ > 1) c2 = *reinterpret_cast<const float4*>(b + ZT + row * W + col);
                        z[0] = k.zc(a.x, c2.x);
                        z[1] = k.zc(a.y, c2.y);
                        z[2] = k.zc(a.z, c2.z);
                        z[3] = k.zc(a.w, c2.w);
                    };
                    T zn[4], zs[4], zt[4];
                    const T (&zc)[4] = zthis;
                    zquad(sn, ty + 1, zn);
                    zquad(sb, ty, zs);
                    zquad(sb, ty + 2, zt);
                    const T zw = zval(sb, ty + 1, col - 1), ze = zval(sb, ty + 1, col + 4);
                    T pv[4][NP];
#pragma unroll
                    for (int q = 0; q < NP; q++) {
                        const float4 pq = *reinterpret_cast<const float4*>(sb + NZ * ZT + q * NCT + ty * TW + 4 * tx);
                        pv[0][q] = pq.x;
                        pv[1][q] = pq.y;
                        pv[2][q] = pq.z;
                        pv[3][q] = pq.w;
                    }
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const T z7[7] = {zc[c], zprev[c], zn[c], zs[c], zt[c], c == 0 ? zw : zc[c - 1],
                                         c == 3 ? ze : zc[c + 1]};
                        if constexpr (RawOperand<K>::value)
                            k.center3((int64_t)i * plane + G.o_own + c, z7, sb[ZT + (ty + 1) * W + col + c], pv[c], acc);
                        else
                            k.center((int64_t)i * plane + G.o_own + c, z7, pv[c], acc);
                    }
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        zprev[c] = zthis[c];
                        zthis[c] = zn[c];
                    }
                }
            }
        }
        cp_async_wait<0>();
        __syncthreads();                        // every plane of this item has been read
        const int next = s_next;                // written before this item's barriers
        Geo GN = G;
        if (next < m.nitems) {
            GN = geometry(next);
            prologue(GN);                       // every plane of this item has been read
        }
        if constexpr (K::Q > 0) {
            double tot[K::Q];
            if (item_reduce<K::Q>(acc, partials, m.item_base + item, m.nitems_total ? m.nitems_total : m.nitems,
                                  &st->count, tot) &&
                tid == 0)
                k.done(st, tot);
        }
        __syncthreads();                        // s_next is rewritten at the next item's start
        item = next;
        G = GN;
    }
    cp_async_wait<0>();
    // the last block out resets the queue for the next launch
    if (tid == 0) {
        const unsigned prev = atomicAdd(&st->exitc, 1u);
        if (prev == gridDim.x - 1) {
            st->queue = 0u;
            st->exitc = 0u;
            __threadfence();
        }
    }
}

// The plane runs of a tile for a kernel with `slots` resident blocks: an item of
// p planes costs a block about p + 3 plane times (filling its pipeline and its
// reduction), and the last round of items is usually not full, so take the
// number of runs whose rounds are the cheapest.  Runs of 4 planes, as many as
// gave four items a block, cost 128^3 steps 2.12 ms and 192^3 steps 5.28; 15-
// and 28-plane runs in two and four rounds 1.78 and 4.68 (1.5 or 5 in place of
// 3 planes: within 4 % either way).  With several field components (stacked
// along i) runs stay inside one.
inline void march_split(const GridDev& g, MarchCfg& m, int64_t slots, int max_items) {
    const int nc = g.ncomp, n0c = g.n[0] / nc;
    const int64_t tiles = (int64_t)m.tiles_x * m.tiles_y * nc;
    int64_t best = 0;
    for (int runs = 1; runs <= n0c; runs++) {
        const int p = (n0c + runs - 1) / runs;
        if (runs > 1 && (p < 4 || tiles * runs > max_items)) break;
        if ((n0c + p - 1) / p != runs) continue;   // the same runs as with fewer
        const int64_t cost = (tiles * runs + slots - 1) / slots * (p + 3);
        if (runs == 1 || cost < best) {
            best = cost;
            m.planes = p;
            m.cpc = runs;
        }
    }
    m.nitems = (int)(tiles * m.cpc);
}

template <class K, int CPT, bool HALO, bool PAIR>
inline int launch_march_k(dare_ctx* ctx, const GridDev& g, const MarchCfg& m0, const K& kern, SolverState* st,
                          double* partials) {
    MarchCfg m = m0;
    const int ic = PAIR ? 16 / (int)sizeof(typename K::type) : m.cpt;   // first interior column of an operand row
    const size_t smem = MarchDepth<typename K::type>::value * march_stage_elems<K>(m.block.x * m.cpt, m.block.y, ic) *
                        sizeof(typename K::type);
    int per_sm = 0;
    DARE_CUDA(ctx, blocks_per_sm((const void*)k_march<K, CPT, HALO, PAIR>, m.block.x * m.block.y, smem, &per_sm));
    int blocks = per_sm * ctx->num_sms;
    if (m.nitems_total == 0) march_split(g, m, blocks, kMaxBlocks);   // (slabs share the slots of their runs)
    if (blocks > m.nitems) blocks = m.nitems;
    launch_pdl(k_march<K, CPT, HALO, PAIR>, dim3(blocks), m.block, smem, ctx->stream, true, g, kern, st, partials, m);
    DARE_LAUNCHED(ctx);
    return DARE_OK;
}

// 16-byte staging (one copy = 16 / sizeof(T) cells): a row length and tile
// width that are multiples of it, enough threads for the operand copies, and
// 16-byte aligned arrays
template <class K, bool HALO>
inline bool march_pairs_ok(const GridDev& g, const MarchCfg& m, const K& kern, int cpt) {
    const int vec = 16 / (int)sizeof(typename K::type);
    const int nt = (int)(m.block.x * m.block.y), tw = (int)m.block.x * cpt, tj = (int)m.block.y;
    bool ok = g.n[2] % vec == 0 && tw % vec == 0 && (tj + 2) * (tw / vec) + 2 * tj <= nt;
    for (int q = 0; q < K::NP; q++) ok = ok && ((uintptr_t)kern.ps[q] & 15) == 0;
    for (int z = 0; z < K::NZ; z++) {
        ok = ok && ((uintptr_t)kern.zs[z] & 15) == 0;
        if (HALO)
            for (int h = 0; h < 2; h++) ok = ok && ((uintptr_t)m.halo[z][h] & 15) == 0;
    }
    return ok;
}

template <class K, int CPT, bool HALO>
inline int launch_march_t(dare_ctx* ctx, const GridDev& g, const MarchCfg& m, const K& kern, SolverState* st,
                          double* partials) {
    if constexpr ((CPT == 1 && sizeof(typename K::type) == 8) || (CPT == 2 && sizeof(typename K::type) == 4)) {
        if (march_pairs_ok<K, HALO>(g, m, kern, CPT))
            return launch_march_k<K, CPT, HALO, true>(ctx, g, m, kern, st, partials);
    }
    return launch_march_k<K, CPT, HALO, false>(ctx, g, m, kern, st, partials);
}

// Two cells per thread (K::kPairs) paid off for steps 1, 2 and 3 while one
// cell per thread staged every value with its own 8-byte copy (256^3: 0.291
// -> 0.257 ms for step 1).  With the 16-byte paired staging of the FP64
// one-cell kernels (PAIR in k_march) one cell per thread is ahead again
// (step 1 0.255 -> 0.252 ms, step 2 0.254 -> 0.249, step 3 0.252 -> 0.249),
// so the FP64 steps run one cell per thread on 32 x 8 tiles; the FP32
// kernels keep two or four cells per thread.  With eight streams and five
// dot products (step 4: 0.316 -> 0.404 ms with two cells), or many outputs
// per cell (init: 0.29 -> 0.38 ms, fold), two cells per thread never paid.
// HALO: the slab variant, which reads m.halo (ignored otherwise).
template <class K, bool HALO = false>
inline int launch_march(dare_ctx* ctx, const GridDev& g, const MarchCfg& m, const K& kern, SolverState* st,
                        double* partials) {
    if (m.nitems > kMaxBlocks || m.item_base + m.nitems > kMaxBlocks || m.nitems_total > kMaxBlocks)
        return set_error(ctx, DARE_ERR_UNSUPPORTED, "grid too large for the reduction");
    if (m.cpt == 4) {   // FP32 grids with n2 a multiple of 4, 64-cell tiles
        if constexpr (sizeof(typename K::type) == 4 && !SplitOperands<K>::value) {
            MarchCfg m2 = m;   // two cells per thread on the same tiles, 16-byte staging
            m2.cpt = 2;
            m2.block = dim3(m.block.x * 2, m.block.y, 1);
            if (march_pairs_ok<K, HALO>(g, m2, kern, 2)) return launch_march_k<K, 2, HALO, true>(ctx, g, m2, kern, st, partials);
            if constexpr (K::kPairs) {
                return launch_march_t<K, 4, HALO>(ctx, g, m, kern, st, partials);
            } else {
                MarchCfg m2 = m;   // two cells per thread on the same tiles
                m2.cpt = 2;
                m2.block = dim3(m.block.x * 2, m.block.y, 1);
                return launch_march_t<K, 2, HALO>(ctx, g, m2, kern, st, partials);
            }
        }
        return set_error(ctx, DARE_ERR_UNSUPPORTED, "four cells per thread are for FP32 kernels");
    }
    if constexpr (K::kPairs) {
        if (m.cpt == 2) return launch_march_t<K, 2, HALO>(ctx, g, m, kern, st, partials);
    }
    if (m.cpt == 1) return launch_march_t<K, 1, HALO>(ctx, g, m, kern, st, partials);
    MarchCfg m1 = m;   // the same tiles, one cell per thread
    m1.cpt = 1;
    m1.block = dim3(m.block.x * m.cpt, m.block.y, 1);
    return launch_march_t<K, 1, HALO>(ctx, g, m1, kern, st, partials);
}

// The scalars of an iteration that the last kernel applies, and one cell of it:
// from the iterate's x, r, u and the products v, s, w, t of steps (6), (9),
// (13), (18)
//   u5 = r - beta5 u (5), r8 = r - alpha1 v (8), x10 = x + alpha1 u5 (10),
//   v12 = s - beta v (12), u15 = r8 - beta u5 (15), r16 = r8 - alpha v12 (16),
//   s17 = s - alpha w (17), then
//   x = x10 + w1 r16 + w2 s17 + alpha u15 (24), r = r16 - w1 s17 - w2 t (25),
//   u = u15 - w1 v12 - w2 w
template <typename T>
struct Step5 {
    T w1, w2, alpha, alpha1, beta, beta5;
    __device__ __forceinline__ explicit Step5(const SolverState* st)
        : w1((T)st->omega1), w2((T)st->omega2), alpha((T)st->alpha), alpha1((T)st->alpha1), beta((T)st->beta),
          beta5((T)st->beta5) {}
    __device__ __forceinline__ void cell(T& x, T& r, T& u, T v, T s, T w, T t) const {
        const T u5 = r - beta5 * u;
        const T r8 = -alpha1 * v + r;
        const T x10 = alpha1 * u5 + x;
        const T v12 = s - beta * v;
        const T u15 = r8 - beta * u5;
        const T r16 = -alpha * v12 + r8;
        const T s17 = -alpha * w + s;
        const T xc = w1 * r16 + w2 * s17 + x10;
        x = alpha * u15 + xc;
        r = -w1 * s17 + -w2 * t + r16;
        u = -w1 * v12 + -w2 * w + u15;
    }
};

// K5: the rest of the iteration (Step5), ||r||, <r_hat_0, r>, then the next
//     iteration's (3), (4).  Eight arrays read, three written.
//     `base` / `total`: partial-sum slots shared with other launches (slabs;
//     0, 0: this launch alone).  `vec4` (FP32 only; n % 4 == 0 and every
//     array 16-byte aligned): four cells per thread and 16-byte accesses
//     (512^3: 0.92 ms; with 4-byte accesses the FP32 kernel took 1.22 ms,
//     81 % of copy bandwidth, both with nine arrays read).
//     In FP64 the products and x, which the next kernels do not read, are
//     loaded and stored as the first to leave L2, so that r, u and rh stay for
//     step 1 (128^3 time step 1.62 -> 1.57 ms, 192^3 4.52 -> 4.48; in FP32 the
//     256^3 refined solve lost 0.4 %).  Two cells a thread and loop trip gave 0.6 %
//     at 256^3 and took the gain at 128^3 away (an odd last trip).
template <typename T>
__device__ __forceinline__ T ld_once(const T* p) {
    if constexpr (sizeof(T) == 8)
        return __ldcs(p);
    else
        return *p;
}
template <typename T>
__device__ __forceinline__ void st_once(T* p, T v) {
    if constexpr (sizeof(T) == 8)
        __stcs(p, v);
    else
        *p = v;
}
template <typename T>
__global__ void __launch_bounds__(256) k_step5(int64_t n, T* __restrict__ x, T* __restrict__ r, T* __restrict__ u,
                                               const T* __restrict__ v, const T* __restrict__ s,
                                               const T* __restrict__ w, const T* __restrict__ t,
                                               const T* __restrict__ rh, SolverState* st, double* partials, int base,
                                               int total, int vec4) {
    pdl_wait();
    pdl_launch();
    if (st->done) return;
    const Step5<T> f(st);
    double acc[2] = {0., 0.};
    if constexpr (sizeof(T) == 4) {
        if (vec4) {
            const int64_t n4 = n >> 2;
            for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n4;
                 q += (int64_t)gridDim.x * blockDim.x) {
                float4 xq = reinterpret_cast<const float4*>(x)[q], rq = reinterpret_cast<const float4*>(r)[q];
                float4 uq = reinterpret_cast<const float4*>(u)[q];
                const float4 vq = reinterpret_cast<const float4*>(v)[q], sq = reinterpret_cast<const float4*>(s)[q];
                const float4 wq = reinterpret_cast<const float4*>(w)[q], tq = reinterpret_cast<const float4*>(t)[q];
                const float4 hq = reinterpret_cast<const float4*>(rh)[q];
                f.cell(xq.x, rq.x, uq.x, vq.x, sq.x, wq.x, tq.x);
                f.cell(xq.y, rq.y, uq.y, vq.y, sq.y, wq.y, tq.y);
                f.cell(xq.z, rq.z, uq.z, vq.z, sq.z, wq.z, tq.z);
                f.cell(xq.w, rq.w, uq.w, vq.w, sq.w, wq.w, tq.w);
                reinterpret_cast<float4*>(x)[q] = xq;
                reinterpret_cast<float4*>(r)[q] = rq;
                reinterpret_cast<float4*>(u)[q] = uq;
                acc[0] += (double)rq.x * (double)rq.x;
                acc[1] += (double)hq.x * (double)rq.x;
                acc[0] += (double)rq.y * (double)rq.y;
                acc[1] += (double)hq.y * (double)rq.y;
                acc[0] += (double)rq.z * (double)rq.z;
                acc[1] += (double)hq.z * (double)rq.z;
                acc[0] += (double)rq.w * (double)rq.w;
                acc[1] += (double)hq.w * (double)rq.w;
            }
            n = 0;   // the scalar loop below has nothing left to do
        }
    }
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        T xc = ld_once(x + c), rc = r[c], uc = u[c];
        f.cell(xc, rc, uc, ld_once(v + c), ld_once(s + c), ld_once(w + c), ld_once(t + c));
        st_once(x + c, xc);
        r[c] = rc;
        u[c] = uc;
        acc[0] += (double)rc * (double)rc;
        acc[1] += (double)rh[c] * (double)rc;
    }
    double tot[2];
    if (!grid_reduce<2>(acc, partials, &st->count, tot, base, total)) return;
    if (threadIdx.x == 0) finish_update(st, tot);
}

// Step (10) of an iteration that stopped after it and before K5 (a
// breakdown in steps (14), (20) or (21)): x = x + alpha1 u of step (5), formed
// from the r and u that K5 has not replaced.
inline __host__ __device__ bool step10_pending_state(int status, int step) {
    return status == ST_TAU0 || (status == ST_BREAKDOWN && (step == 14 || step == 20));
}
template <typename T>
__global__ void k_step10(int64_t n, const SolverState* st, const T* __restrict__ r, const T* __restrict__ u,
                         T* __restrict__ x) {
    if (!step10_pending_state(st->status, st->step)) return;   // read on the device: no host round trip
    const T alpha1 = (T)st->alpha1, beta5 = (T)st->beta5;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const T u5 = r[c] - beta5 * u[c];
        x[c] = alpha1 * u5 + x[c];
    }
}
inline bool step10_pending(const SolverState& st) { return step10_pending_state(st.status, st.step); }


static __global__ void k_invdiag(const double* __restrict__ dc, double* __restrict__ invd, int64_t n) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
        invd[c] = 1. / dc[c];
}

// x = invd .* x (applyRightPrec at the end of the solve)
static __global__ void k_scale(int64_t n, const double* __restrict__ invd, double* __restrict__ x) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
        x[c] = invd[c] * x[c];
}

}  // namespace dare_gpu
