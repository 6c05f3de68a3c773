// Host-side launch interface of the residual-and-update kernels.
#pragma once

#include "solver.cuh"

namespace ccfd {

// Launch whose CTAs may be set up while the kernel before it on the stream
// drains (programmatic dependent launch); they wait in grid_wait(), first
// thing and on every path, so completion stays in stream order.  Microseconds
// per stage without / with: 8,000 cells 14.15 / 13.65, 32,761 cells 15.15 /
// 14.60, 500,000 cells 77.8 / 77.0.  The kernels do not release their
// dependents early: waiting CTAs then take the slots of running ones (16.6 us
// at 8,000 cells).
template <typename... P, typename... A>
inline void launch_dependent(void (*kern)(P...), dim3 grid, int threads, int smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, args...);
}
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Tiles of the flux kernel in device memory (see tiles.h): tile t owns the
// cells [t * cells, (t + 1) * cells) and evaluates every face that touches
// them.  Faces are numbered tile by tile, each by the first tile that touches
// it: a tile's own faces are consecutive, the others are listed.
struct TileDev {
    int n_tiles;
    int cells;            // cells per tile
    int max_f;            // most faces of a tile (its shared-memory flux buffer)
    int threads;          // CTA size of the flux kernel (0: the precision's default)
    const int4* rng;      // [n_tiles] (first own face, own faces, first border entry, border entries)
    const int* border;    // faces of earlier tiles
    const double4* f_nl;  // [F] (n.x, n.y, len, owner cell | neighbour cell or -1-g as two words)
    const double4* f_gp;  // [F] face midpoint minus the barycentre of the owner / neighbour (Navier-Stokes)
    const double4* f_bb;  // [F] (baryBaryVec.x, .y, baryBaryDist, 0) (Navier-Stokes)
    const int2* g_rng;    // [n_tiles] (first entry, entries) of the tile's ghosts
    const int4* ghost;    // [B] by tile: ghost, its cell, slot of its face's owner state, 0
    const ushort4* u_code;  // [N] per side 2 * local face + neighbour flag, 0xffff padded
};

// Per-ghost data of the boundary code (device order of ghosts = BCside order).
struct GhostDev {
    const int* bc;         // BC table index
    const double4* gn;     // (ghost bary x, y, n.x, n.y)
    const double2* mid;    // face midpoint
    double4* state;        // [B] state at the mirrored barycentre (written by k_grad)
    double4* face;         // [B] state at the boundary face (written by k_grad)
};

// One residual evaluation (optionally fused with a Runge-Kutta stage).
struct alignas(16) StageLaunch {
    DevMesh mesh;
    TileDev tiles;
    GhostDev ghosts;
    Gas gas;
    const Phys* phys_g;    // all physics constants in global memory (boundary code)
    StepParams sp;
    const Ctrl* ctrl;      // device control block, or nullptr (fixed time)
    double tfix;           // time when ctrl == nullptr
    double a_time;         // stage time = t + a_time * dt
    int order, limiter, flux_id, ns;
    int fp32;              // 1: FP32 reconstruction and face fluxes (mixed precision)
    int mode;              // 0: residual u_t only; 1: RK stage
    const int* skip;       // batched residual evaluations: skipped while *skip != 0
    const double4* prim_in;
    double4* prim_out;     // RK: updated primitive state
    double4* prim_buf[2];  // batched RK stages: the two state buffers (prim_in / prim_out by parity and stage)
    double4* cons0;        // RK: stage-start conservative state (updated in place at the last stage)
    double* ghost_pface;   // [B] interior face pressure at boundary faces
    double4* u_t;          // [N] residual (mode 0, or RK last stage), may be nullptr
    void* grad;            // [2N] limited gradients (Navier-Stokes), double4 or float4 (fp32)
    void* fstate;          // [2F] reconstructed states at the faces (Euler, second order), likewise
    double4* grad_out;     // [2N] limited gradients for the caller, may be nullptr
    double rk;
    int last_stage;
    double* res_partial;   // [4 * n_tiles] or nullptr
    double2* dt_partial;   // [n_tiles] (last RK stage) or nullptr
    int* dt_bad;           // [n_tiles]
    unsigned* flags;
    unsigned* ticket;      // CTA completion counter of the last stage (zero between launches)
    const int* wall_ghost; // wing surface ghosts in calcCoef summation order
    const double* wall_nl; // their (n.x, n.y, len)
};

// One launch over the concatenated tiles of several instances that share the
// kernel variant (flux, order, equations, precision).
struct BatchLaunch {
    const StageLaunch* recs;  // one per instance
    const int4* tmap;         // [n_tiles] (instance, tile, control block or skip word address)
    int n_tiles, smem_bytes;
    int rk_mode, stage;
    int flux_id, order, ns, fp32;
};

// entry of a batch's tile map: `word` is the instance's control block (RK
// stages) or its skip word (residual evaluations), so that a CTA reads it
// together with the instance's record
inline int4 tile_entry(int inst, int tile, const void* word) {
    const unsigned long long p = (unsigned long long)word;
    return make_int4(inst, tile, (int)(unsigned)(p & 0xffffffffu), (int)(unsigned)(p >> 32));
}

void launch_stage(const StageLaunch& L, cudaStream_t st);
void launch_stage_batch(const BatchLaunch& B, cudaStream_t st);
// The gradient kernel alone.  It writes the limited gradients to L.grad_out if
// that is set, the reconstructed face states (Euler, L.fstate) or the gradients
// (Navier-Stokes, L.grad), the ghost states at the barycentres and the boundary
// faces, and, if L.ghost_pface is set, the wall pressures.
void launch_gradients(const StageLaunch& L, cudaStream_t st);
// dynamic shared memory of a batched flux launch over tiles of up to max_f faces
int stage_smem_bytes(int max_f, int fp32);
void launch_dt(const DevMesh& m, const Gas& P, const Ctrl* ctrl, const StepParams& sp,
               const double4* prim, double2* partial, int* bad_partial, cudaStream_t st);
void launch_step_begin(Ctrl* ctrl, const StepParams& sp, const double2* partial,
                       const int* bad_partial, int nb, cudaStream_t st);
int error_blocks(int n_cells);
void launch_exact_state(int n, const double4* xq, const Phys* phys_g, int which, double time, double4* out,
                        unsigned* flags, cudaStream_t st);
void launch_errors(const DevMesh& m, const double4* xq, const double4* prim, const double4* grad,
                   const Phys* phys_g, int which, double time, double* partial, unsigned* flags,
                   cudaStream_t st);
void imp_step_end_launch(Ctrl* ctrl, const DevMesh& m, const Gas& P, const StepParams& sp,
                         const double* res_partial, int nres, double2* dt_partial, int* dt_bad, int ndt,
                         const int* wall_ghost, const double* wall_nl, const double* ghost_pface,
                         const double4* prim_new, cudaStream_t st);

}  // namespace ccfd
