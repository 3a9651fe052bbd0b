// dare_internal.cuh -- shared types and helpers of the sm_100a implementation.
//
// Memory layout in HBM (one B200 holds a 512^3 FP64 system):
//   * fields: ghosted arrays, (nx+2g)(ny+2g)(nz+2g) doubles per time level,
//     last dimension fastest (Data/GridVector.inl:68-71 with N = 1);
//   * system: structure-of-arrays diagonals diag[slot][cell], slot order
//     CENTER, WEST, EAST, SOUTH, NORTH, BOTTOM, TOP, plus rhs and x, all over
//     internal cells only (the Tpetra row map, Trilinos.inl:467-504);
//   * solver work vectors over internal cells; scalars live on the device.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/dare_gpu.h"

namespace dare_gpu {

constexpr int kSlots = 7;

struct GridDev {             // passed by value to kernels
    int dim;
    int ng;
    int n[3];                 // internal resolution (1 when inactive)
    int gn[3];                // ghosted resolution
    int og[3];                // ghost offset per dimension (0 when inactive)
    int periodic[3];
    int64_t ncell;
    int64_t ncell_ghosted;
    double dx[3];
    double volume;
    double area[3];
    // Staggered representation (CartesianRepresentation.inl:33-76): one more
    // cell along a staggered, non-periodic direction, the cell width of the
    // base grid, and the domain starting half a cell earlier (origin = -dx/2;
    // 0 otherwise).
    int staggered[3];
    double origin[3];
    // Solver view of a system with several field components: the components
    // are stacked along i (n[0] = ncomp x the grid's n0, ncell likewise), each
    // component's planes wrapping among themselves on a periodic x.
    int ncomp = 1;
};

}  // namespace dare_gpu

namespace dare_gpu {
// kernel ids for the optional per-kernel event timing
enum KernelId : int {
    KID_ASSEMBLE = 0,
    KID_FOLD = 1,
    KID_INIT = 2,
    KID_STEP1 = 3,
    KID_STEP2 = 4,
    KID_STEP3 = 5,
    KID_STEP4 = 6,
    KID_STEP5 = 7,
    KID_SOLVE = 8,   // the whole solve of a small system (dare_resident.cu)
    KID_COUNT = 16
};
}  // namespace dare_gpu

struct dare_ctx {
    int device = 0;
    int num_sms = 148;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    std::string last_error;
    int64_t launches = 0;
    // waits between the blocks of a one-launch solve (dare_ctx_set_wait_limit,
    // dare_ctx_debug_give_up)
    int team_polls = 0, debug_quitter = -1;
    // the most blocks of a one-launch solve, in one cluster and over the device
    // (dare_ctx_set_team_blocks; negative: what the device holds)
    int team_cluster = -1, team_grid = -1;
    // Streams beside `stream`, with their events, made when something first runs
    // side by side (ensure_side): the cluster sizes of a batch, the lanes of a
    // network's minibatch.  A batch of one small box took 0.58 ms to make and
    // destroy with five streams of its own, 0.36 without.
    cudaStream_t side[5] = {nullptr};
    cudaEvent_t fork = nullptr, join[5] = {nullptr};
    int box_classes = -1;   // cluster sizes the device holds (dare_batched.cu; -1: not asked yet)
    // per-kernel CUDA-event timing (dare_ctx_set_profiling)
    int profiling = 0;
    cudaEvent_t ev[16] = {nullptr};
    double stat_ms[dare_gpu::KID_COUNT] = {0};
    int64_t stat_n[dare_gpu::KID_COUNT] = {0};
};

struct dare_grid {
    dare_ctx* ctx = nullptr;
    dare_gpu::GridDev dev{};
};

// Every handle records its device at creation: its destroy function uses
// that, never the context or grid it was made from, so handles may be
// destroyed in any order (a garbage collector's, for instance).
struct dare_field {
    dare_grid* grid = nullptr;
    int device = 0;
    int num_levels = 0;
    int ncomp = 1;                // components, stored component-major: level[l][c * ncell_ghosted + cell]
    double* level[8] = {nullptr};
};

struct dare_solver_ws;  // defined in dare_bicgstab2.cu
void dare_solver_ws_free(dare_solver_ws* ws);

struct dare_system {
    dare_grid* grid = nullptr;
    int device = 0;
    int ncomp = 1;               // field components (block-diagonal, one 7-point stencil each)
    dare_gpu::GridDev sdev{};    // the solver's view: components stacked along i
    int bc_type[6] = {0, 0, 0, 0, 0, 0};        // the faces' conditions of every component ...
    double bc_value[6] = {0, 0, 0, 0, 0, 0};
    // ... unless a component has its own (dare_system_set_bc_component):
    // per component, 6 faces each; empty until the first per-component call
    std::vector<int> bc_type_c;
    std::vector<double> bc_value_c;
    // A slab of a larger grid (dare_slabs.cu): x ends shared with a
    // neighbouring slab (bit 0 low, bit 1 high), whose faces are not folded.
    int xint = 0;
    double* diag = nullptr;   // [7][ncomp][ncell], component-major within a slot
    double* rhs = nullptr;    // [ncomp][ncell]
    double* x = nullptr;
    dare_solver_ws* ws = nullptr;
};

namespace dare_gpu {

// ---- error handling: never abort, record the message on the context ------
int set_error(dare_ctx* ctx, int code, const std::string& msg);
int check_cuda(dare_ctx* ctx, cudaError_t e, const char* what);
#define DARE_CUDA(ctx, call)                                              \
    do {                                                                   \
        cudaError_t _e = (call);                                           \
        if (_e != cudaSuccess) return ::dare_gpu::check_cuda(ctx, _e, #call); \
    } while (0)
#define DARE_LAUNCHED(ctx)                                                 \
    do {                                                                   \
        (ctx)->launches++;                                                 \
        cudaError_t _e = cudaGetLastError();                               \
        if (_e != cudaSuccess) return ::dare_gpu::check_cuda(ctx, _e, "kernel launch"); \
    } while (0)

// ---- index helpers -------------------------------------------------------
__host__ __device__ inline int64_t local_index(const GridDev& g, int i, int j, int k) {
    return ((int64_t)(i + g.og[0]) * g.gn[1] + (j + g.og[1])) * g.gn[2] + (k + g.og[2]);
}

// Neighbour ordinal in the internal numbering, wrapped on periodic
// dimensions; a removed (non-periodic boundary) or inactive neighbour maps to
// the cell itself so every access stays in bounds (its coefficient is 0).
__host__ __device__ inline void neighbour_ordinals(const GridDev& g, int i, int j, int k, int64_t c,
                                                    int64_t nb[7]) {
    const int64_t sx = (int64_t)g.n[1] * g.n[2], sy = g.n[2];
    nb[0] = c;
    nb[1] = i > 0 ? c - sx : (g.periodic[0] ? c + (int64_t)(g.n[0] - 1) * sx : c);
    nb[2] = i < g.n[0] - 1 ? c + sx : (g.periodic[0] ? c - (int64_t)(g.n[0] - 1) * sx : c);
    nb[3] = j > 0 ? c - sy : (g.periodic[1] ? c + (int64_t)(g.n[1] - 1) * sy : c);
    nb[4] = j < g.n[1] - 1 ? c + sy : (g.periodic[1] ? c - (int64_t)(g.n[1] - 1) * sy : c);
    nb[5] = k > 0 ? c - 1 : (g.periodic[2] ? c + (g.n[2] - 1) : c);
    nb[6] = k < g.n[2] - 1 ? c + 1 : (g.periodic[2] ? c - (g.n[2] - 1) : c);
}

// ---- programmatic dependent launch ----------------------------------------
// Kernels of the network and of the solver's iterations follow one another
// every 3-50 us.  Launched this way, a kernel's blocks may be placed while the
// one before it still runs; they meet it at pdl_wait(), which every thread
// passes before it touches anything that an earlier kernel writes, and which
// ends when the earlier kernel has ended and its stores are visible.  Only
// then do they let the next kernel in (pdl_launch): so when a kernel's first
// instructions run, every kernel but the one directly before it is complete,
// and what those wrote (the convolutions' weights) may be read ahead of the
// wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A launch that need not wait for the kernel before it to end (`overlap` off:
// an ordinary one)
template <typename... P, typename... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool overlap,
                       A&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = at;
    c.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);   // an error is picked up by DARE_LAUNCHED
}

// The blocks of a kernel that an SM of the current device holds (at least 1), with
// its limit of dynamic shared memory raised to `smem`.  The limit belongs to the
// kernel on its device, for every context, system and thread alike, and is only
// ever raised, so that no launch is refused because another one needed less.
cudaError_t blocks_per_sm(const void* kernel, int threads, size_t smem, int* blocks);

// Side stream q of a context, its event and the one the side streams start from
int ensure_side(dare_ctx* ctx, int q);

inline int grid_blocks(const dare_ctx* ctx, int64_t work, int threads, int per_sm) {
    int64_t b = (work + threads - 1) / threads;
    int64_t cap = (int64_t)ctx->num_sms * per_sm;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

}  // namespace dare_gpu
