// Implicit backward-Euler path: Newton iteration with matrix-free GMRES and
// the LU-SGS preconditioner.
//
//   implicitTimeStep  src/timeDiscretization.c:412-552
//   GMRES_M           src/linearSolver.c:385-510 (right-preconditioned, one
//                     cycle of nKdim, modified Gram-Schmidt, Givens rotations)
//   matrixVector      src/linearSolver.c:343-373 (finite-difference Jacobian
//                     product (v - alpha dt (R(X + eps v) - R(X)) / eps),
//                     eps = sqrt(DBL_EPSILON) / |v|)
//   buildMatrix       src/linearSolver.c:186-252 (finite-difference Jacobian
//                     with respect to the primitive variables, diagonal and
//                     face-neighbour 4x4 blocks only, I - dt J)
//   calcDinv          src/linearSolver.c:136-179 (4x4 inverse, singular when
//                     |det| <= DBL_EPSILON)
//   LUSGS             src/linearSolver.c:261-333 (forward / backward sweeps in
//                     the reference's cell numbering)
//
// The reference stores the Jacobian densely, (4N)^2 doubles, and builds it
// with 4N residual evaluations.  Here the same entries live in block-sparse
// storage (one 4x4 block per cell and one per half-side) and the columns are
// obtained with 4 residual evaluations per colour of a distance-3 colouring:
// cells of one colour are far enough apart that their perturbations reach
// disjoint sets of recorded residuals.  The sweeps are level-scheduled: a
// cell's level is one more than the highest level among its neighbours of
// lower (forward) / higher (backward) reference number, so every level is a
// set of independent cells and the sweep result is exactly the sequential
// one.
//
// Every kernel works on a set of members (independent cases) at once:
// blockIdx.y selects the member's descriptor, blockIdx.x the block of its
// cells.  All members advance in lockstep through the same sequence of
// Newton and Krylov iterations; a member whose GMRES cycle or Newton loop has
// ended (or failed) is switched off by flags in device memory and its blocks
// return at once, so the result of every member is exactly that of the
// member running alone.  A single case is a set of one.
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <thread>
#include <tuple>
#include <vector>

#include "ccfd_ctx.cuh"
#include "colouring.h"
#include "host/ccfd_host.h"
#include "kernels.cuh"

using namespace ccfd;

namespace {

constexpr int kB = 256;  // threads per block of the vector kernels
constexpr int kSweepThreads = 512;  // threads of the LU-SGS CTA (one per member), 4 per cell

// device scalars of one implicit step (offsets into ImpState::sc)
enum Sc {
    SC_NORMB = 0, SC_ABORT, SC_EPSFD, SC_NORM_X0, SC_NORM_XK, SC_EPS2LOC, SC_TMP,
    SC_H = 16
};

// per-member control words (ImpDev::ctl)
enum Ctl {
    CTL_NEWTON = 0,    // Newton loop of the current time step running
    CTL_INNER,         // Newton iterations of the current time step
    CTL_GMRES_TOTAL,   // GMRES iterations so far (report)
    CTL_NEWTON_TOTAL,  // Newton iterations so far (report)
    CTL_SKIP_JAC,      // residual evaluations of the Jacobian colour loop skipped
    CTL_STATUS,        // failure status (ccfd_status) of the current step
    CTL_SKIP_NEWTON,   // == !CTL_NEWTON (skip word of the Newton residuals)
    CTL_SKIP_GMRES,    // GMRES iteration skipped (cycle ended or Newton off)
    CTL_WORDS = 8
};

struct SweepRec;

// Device descriptor of one member (pointers into its context and state).
struct ImpDev {
    long N;
    int K, nb, precond, n_newton;
    double gam1, eps_gmres, eps2newton;
    double4 *XK, *Q, *RXK, *F, *dX, *W, *V, *Z, *ptmp, *ut, *dxs, *cons, *prim;
    double4 *pert[4], *utj[4];  // Jacobian columns: perturbed states and their residuals, one per variable
    double *D, *Dinv, *O, *sc, *partial;
    // mixed precision (fp32 = 1): Krylov basis V, Z, the sweep vector and the
    // LU-SGS blocks D^-1, O in FP32 (Vf, Zf, dxsf, Dinvf, Of instead of the
    // FP64 arrays); residuals, W, the Newton update and GMRES scalars FP64
    int fp32;
    float4 *Vf, *Zf, *dxsf;
    float *Dinvf, *Of;
    double4* rjb;  // mixed precision: R(U, t) of the FP32-flux evaluation, base of the Jacobian columns
    int* flag;  // [0] GMRES cycle done, [1] final m, [2] singular, [3] non-finite, [4] a sweep gave up
    int* ctl;   // Ctl words
    Ctrl* ctrl;
    const int *hs_off, *hs_nb, *twin;
    int ncol;
    const int *color_off, *color_cells;
    int n_lev_f, n_lev_b;
    // sweeps in level order: level offsets; per position the cell, its
    // lower (forward) / upper (backward) neighbours and the half-sides of
    // their off-diagonal blocks in side order, -1 padded to four
    const int *lev_f_off, *fw_cell, *lev_b_off, *bw_cell;
    const int4 *fw_nb, *fw_h, *bw_nb, *bw_h;
    // forward / backward sequences of the cluster kernel's warps: chunk
    // offsets [kClWorkers + 1], records (8 per chunk)
    const int* cl_off[2];
    const SweepRec* cl_rec[2];
};

struct ImpState {
    int K = 0;            // nKdim
    long N = 0;
    double4 *XK = nullptr, *Q = nullptr, *RXK = nullptr, *F = nullptr, *dX = nullptr;
    double4 *W = nullptr, *V = nullptr, *Z = nullptr, *ptmp = nullptr, *ut = nullptr;
    double4 *dxs = nullptr;
    double *D = nullptr, *Dinv = nullptr, *O = nullptr;  // [N][16], [N][16], [H][16]
    bool fp32 = false;           // mixed precision: the FP32 arrays below instead
    float4 *Vf = nullptr, *Zf = nullptr, *dxsf = nullptr;
    float *Dinvf = nullptr, *Of = nullptr;
    double4* RJB = nullptr;      // mixed precision: base residual of the Jacobian columns
    // the four columns of a colour, evaluated by the same launches: state,
    // residual, reconstruction and ghost scratch of each
    double4 *jpert[4] = {}, *jut[4] = {}, *jghost[4] = {};
    void* jrec[4] = {};
    double* sc = nullptr;        // device scalars
    int* flag = nullptr;         // [0] gmres done, [1] m_final, [2] singular, [3] non-finite
    int* ctl = nullptr;          // Ctl words
    double* partial = nullptr;   // per-block partial sums, two buffers of nb + 1
    int nb = 0;
    // colouring (device cell lists per colour) and neighbour twins
    std::vector<int> color_off;  // host copy of the colour offsets
    int* color_off_d = nullptr;
    int* color_cells = nullptr;
    int* twin = nullptr;         // [H] half-side of the neighbour that points back
    // LU-SGS level schedules
    int n_lev_f = 0, n_lev_b = 0;
    int *lev_f_off = nullptr, *fw_cell = nullptr, *lev_b_off = nullptr, *bw_cell = nullptr;
    int4 *fw_nb = nullptr, *fw_h = nullptr, *bw_nb = nullptr, *bw_h = nullptr;
    bool cluster_ok = false;     // the sweeps fit the cluster kernel
    int* cl_off[2] = {nullptr, nullptr};
    SweepRec* cl_rec[2] = {nullptr, nullptr};
    bool ready = false;
    void* solo = nullptr;        // the member set of this context running alone
    std::vector<int> hs_off_h;   // device CSR offsets of the half-sides (host copy)
    bool jac_built = false;      // ccfd_build_matrix has filled the blocks
};

__device__ __forceinline__ void ld(const double4& v, double q[4]) {
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
}
__device__ __forceinline__ double4 mk(const double q[4]) { return make_double4(q[0], q[1], q[2], q[3]); }

// per-cell a.b with the reference's term order (src/linearSolver.c:121-124)
__device__ __forceinline__ double cell_dot(const double4& a, const double4& b) {
    double r = 0.0;
    r += a.x * b.x;
    r += a.y * b.y;
    r += a.z * b.z;
    r += a.w * b.w;
    return r;
}

__device__ __forceinline__ void block_partial(double v, double* partial) {
    __shared__ double sh[32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double x = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) partial[blockIdx.x] = x;
    }
}

// Sum of a member's nb block partials, the same in every block that asks for
// it (kB threads, fixed order).
__device__ __forceinline__ double block_total(const double* partial, int nb) {
    __shared__ double sh[kB];
    double v = 0.0;
    for (int k = threadIdx.x; k < nb; k += kB) v += partial[k];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = kB / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

// A dot product in the kernel that needs it: up to kFusedParts partials are
// summed there by every block, instead of waiting for a launch in between;
// kb_total leaves the sum of more behind them (what every block reads grows
// with the square of the mesh).  Milliseconds of an unpreconditioned step of 12
// to 16 Krylov iterations, summed in the consumers / by kb_total: 32,768 cells
// 1.65 / 1.96, 131,072 2.07 / 2.20, 262,144 2.82 / 3.15, 524,288 (2,048
// partials) 4.17 / 4.12, 1,048,576 7.18 / 6.70, 2,097,152 14.0 / 12.6, 4,194,304
// 27.0 / 21.3.
constexpr int kFusedParts = 2048;
__device__ __forceinline__ double dot_total(const double* partial, int nb) {
    return nb > kFusedParts ? partial[nb] : block_total(partial, nb);
}

// Krylov basis access in the member's precision (FP64 arithmetic outside)
__device__ __forceinline__ double4 getV(const ImpDev& d, long k) {
    if (d.fp32) {
        float4 v = d.Vf[k];
        return make_double4(v.x, v.y, v.z, v.w);
    }
    return d.V[k];
}
__device__ __forceinline__ double4 getZ(const ImpDev& d, long k) {
    if (d.fp32) {
        float4 v = d.Zf[k];
        return make_double4(v.x, v.y, v.z, v.w);
    }
    return d.Z[k];
}
__device__ __forceinline__ void putV(const ImpDev& d, long k, double4 v) {
    if (d.fp32) d.Vf[k] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    else d.V[k] = v;
}
__device__ __forceinline__ void putZ(const ImpDev& d, long k, double4 v) {
    if (d.fp32) d.Zf[k] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    else d.Z[k] = v;
}

__device__ __forceinline__ bool newton_on(const ImpDev& d) { return d.ctl[CTL_NEWTON] != 0; }
__device__ __forceinline__ bool gmres_on(const ImpDev& d) { return d.ctl[CTL_SKIP_GMRES] == 0; }

// a member's step fails: its Newton loop and GMRES cycle stop, the control
// block records the error and the member does not step again
__device__ void fail_member(const ImpDev& d, int status, unsigned devflag) {
    d.ctl[CTL_STATUS] = status;
    d.ctl[CTL_NEWTON_TOTAL] += d.ctl[CTL_INNER];
    d.ctl[CTL_NEWTON] = 0;
    d.ctl[CTL_SKIP_NEWTON] = 1;
    d.ctl[CTL_SKIP_GMRES] = 1;
    d.flag[0] = 1;
    d.ctrl->flags |= devflag;
    d.ctrl->done = 1;
    d.ctrl->active = 0;
}

// (every kernel of the Newton and Krylov loops is a dependent launch: the
// vector kernels are a few microseconds each; implicit airfoil steps of 32,768
// cells 9.83 -> 9.51 ms a pass of two)
#define MEMBER \
    grid_wait();  \
    const ImpDev& d = I[blockIdx.y]
#define CELL_INDEX                                           \
    if ((int)blockIdx.x >= d.nb) return;                     \
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x

// start of a time step: members whose control block lets them step run
// their Newton loop
__global__ void kb_step_prepare(const ImpDev* __restrict__ I) {
    MEMBER;
    if (threadIdx.x) return;
    int on = d.ctrl->active != 0;
    d.ctl[CTL_NEWTON] = on;
    d.ctl[CTL_SKIP_NEWTON] = !on;
    d.ctl[CTL_SKIP_GMRES] = 1;
    d.ctl[CTL_INNER] = 0;
    d.ctl[CTL_STATUS] = 0;
}

// Q = cVar; pVar = consPrim(cVar) (src/timeDiscretization.c:420-433)
__global__ void kb_step_begin(const ImpDev* __restrict__ I) {
    MEMBER;
    if (!newton_on(d)) return;
    CELL_INDEX;
    if (i >= d.N) return;
    double c[4], p[4];
    double4 cv = d.cons[i];
    d.Q[i] = cv;
    ld(cv, c);
    cons_prim(d.gam1, c, p);
    d.prim[i] = mk(p);
}

// F = (cVar - Q) - alpha dt u_t and its dot partial; at the step start also
// XK = cVar (src/timeDiscretization.c:439-449, 533-536)
__global__ void kb_newton_F(const ImpDev* __restrict__ I, int copy_xk) {
    MEMBER;
    if (!newton_on(d)) return;
    CELL_INDEX;
    double v = 0.0;
    if (i < d.N) {
        const double adt = 1.0 * d.ctrl->dt;
        double c[4], q[4], u[4], f[4];
        double4 cv = d.cons[i];
        ld(cv, c);
        ld(d.Q[i], q);
        ld(d.RXK[i], u);
#pragma unroll
        for (int k = 0; k < 4; ++k) f[k] = c[k] - q[k] - adt * u[k];
        double4 fv = mk(f);
        d.F[i] = fv;
        if (copy_xk) d.XK[i] = cv;
        v = cell_dot(fv, fv);
    }
    block_partial(v, d.partial);
}

// |F|^2 of the Newton loop: into SC_NORM_X0 (first) or SC_NORM_XK
__global__ void kb_newton_norm(const ImpDev* __restrict__ I, int first) {
    MEMBER;
    if (!newton_on(d)) return;
    const double r = block_total(d.partial, d.nb);
    if (threadIdx.x == 0) d.sc[first ? SC_NORM_X0 : SC_NORM_XK] = r;
}

// eps2newtonLoc and the first test of the Newton loop
// (src/timeDiscretization.c:469-478)
__global__ void kb_newton_start(const ImpDev* __restrict__ I) {
    MEMBER;
    if (threadIdx.x || !newton_on(d)) return;
    double n0 = d.sc[SC_NORM_X0];
    double eps2loc = fmax(1e-8 * 1e-8 * d.N * d.eps2newton / n0, d.eps2newton);
    d.sc[SC_EPS2LOC] = eps2loc;
    d.sc[SC_NORM_XK] = n0;
    if (!((n0 > eps2loc * n0) && (0 < d.n_newton))) {
        d.ctl[CTL_NEWTON] = 0;
        d.ctl[CTL_SKIP_NEWTON] = 1;
        if (d.n_newton == 0) {
            d.ctl[CTL_STATUS] = CCFD_ERR_NEWTON;
            d.ctrl->flags |= FLAG_NEWTON;
            d.ctrl->done = 1;
            d.ctrl->active = 0;
        }
    }
}

// GMRES set-up: normB = sqrt(|F|^2), abortCrit, gam[0]; R0 = -B, delX = 0,
// V0 = R0 / normR0 (src/linearSolver.c:385-408)
__global__ void kb_gmres_init(const ImpDev* __restrict__ I) {
    MEMBER;
    if (!newton_on(d)) return;
    CELL_INDEX;
    const double nr = sqrt(d.sc[SC_NORM_XK]);
    if (i == 0) {
        double* H = d.sc + SC_H;
        double* gam = H + (d.K + 1) * (d.K + 1);
        d.sc[SC_NORMB] = nr;
        d.sc[SC_ABORT] = d.eps_gmres * nr;
        gam[0] = nr;
    }
    if (i >= d.N) return;
    double b[4], v[4];
    ld(d.F[i], b);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = -b[k] / nr;
    putV(d, i, mk(v));
    d.dX[i] = make_double4(0.0, 0.0, 0.0, 0.0);
}

// flags of a new GMRES cycle (after kb_gmres_init has run on every block)
__global__ void kb_gmres_flags(const ImpDev* __restrict__ I) {
    MEMBER;
    if (threadIdx.x) return;
    int on = newton_on(d);
    d.flag[0] = on ? 0 : 1;
    d.flag[1] = d.flag[2] = d.flag[3] = d.flag[4] = 0;
    d.ctl[CTL_SKIP_GMRES] = !on;
}

// Z_m = V_m when the preconditioner is off
__global__ void kb_copy_vz(const ImpDev* __restrict__ I, int m) {
    MEMBER;
    if (d.precond || !gmres_on(d)) return;
    CELL_INDEX;
    if (i < d.N) putZ(d, (long)m * d.N + i, getV(d, (long)m * d.N + i));
}

// sums of more than kFusedParts partials of buffer `buf`, left behind them
__global__ void kb_total(const ImpDev* __restrict__ I, int buf) {
    MEMBER;
    if (d.nb <= kFusedParts || !gmres_on(d)) return;
    double* const partial = d.partial + buf * (d.nb + 1);
    const double r = block_total(partial, d.nb);
    if (threadIdx.x == 0) partial[d.nb] = r;
}

// |Z_m|^2 partials; also clears the count of members that iterate on
// (kb_givens counts them)
__global__ void kb_dot_zz(const ImpDev* __restrict__ I, int m, int* count) {
    MEMBER;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *count = 0;
    if (!gmres_on(d)) return;
    CELL_INDEX;
    double v = 0.0;
    if (i < d.N) {
        double4 z = getZ(d, (long)m * d.N + i);
        v = cell_dot(z, z);
    }
    block_partial(v, d.partial);
}

// eps = sqrt(DBL_EPSILON) / |Z_m|; U = XK + eps v, pVar = consPrim(U)
// (src/linearSolver.c:343-360)
__global__ void kb_mv_prep(const ImpDev* __restrict__ I, int m) {
    MEMBER;
    if (!gmres_on(d)) return;
    CELL_INDEX;
    const double e = sqrt(DBL_EPSILON) / sqrt(dot_total(d.partial, d.nb));
    if (i == 0) d.sc[SC_EPSFD] = e;
    if (i >= d.N) return;
    double x[4], z[4], c[4], p[4];
    ld(d.XK[i], x);
    ld(getZ(d, (long)m * d.N + i), z);
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = x[k] + e * z[k];
    cons_prim(d.gam1, c, p);
    d.ptmp[i] = mk(p);
}

// W = v - alpha dt (u_t - R_XK) / eps (src/linearSolver.c:364-372), and the
// partial of the first Gram-Schmidt product V0 . W
__global__ void kb_mv_finish(const ImpDev* __restrict__ I, int m) {
    MEMBER;
    if (!gmres_on(d)) return;
    CELL_INDEX;
    double dd = 0.0;
    if (i < d.N) {
        const double adt = 1.0 * d.ctrl->dt;
        double z[4], u[4], r[4], w[4];
        ld(getZ(d, (long)m * d.N + i), z);
        ld(d.ut[i], u);
        ld(d.RXK[i], r);
        double e = d.sc[SC_EPSFD];
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = z[k] - adt * (u[k] - r[k]) / e;
        double4 wv = mk(w);
        d.W[i] = wv;
        dd = cell_dot(getV(d, i), wv);
    }
    block_partial(dd, d.partial);
}

// H[nn][m] from the partials of V_nn . W; W -= H[nn][m] V_nn (modified
// Gram-Schmidt step, src/linearSolver.c:440-450), then the partial of
// V_{nn+1} . W (or W . W after the last one) into the other partial buffer
// (a member's later blocks may still read this one).  On 32,768 cells a launch
// in between for the sum took 4.6 us of the pair's 10.1, this one takes 6.7.
__global__ void kb_mgs(const ImpDev* __restrict__ I, int nn, int m) {
    MEMBER;
    if (!gmres_on(d)) return;
    CELL_INDEX;
    double* const in = d.partial + (nn & 1) * (d.nb + 1);
    double* const out = d.partial + ((nn + 1) & 1) * (d.nb + 1);
    const double hh = dot_total(in, d.nb);
    if (i == 0) d.sc[SC_H + nn * (d.K + 1) + m] = hh;
    double dd = 0.0;
    if (i < d.N) {
        double w[4], p[4];
        ld(d.W[i], w);
        ld(getV(d, (long)nn * d.N + i), p);
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] -= hh * p[k];
        double4 wv = mk(w);
        d.W[i] = wv;
        dd = nn < m ? cell_dot(getV(d, (long)(nn + 1) * d.N + i), wv) : cell_dot(wv, wv);
    }
    block_partial(dd, out);
}

// H[m+1][m] = |W|, Givens rotations, residual estimate and stop test of
// iteration m, and the back substitution when the cycle ends
// (src/linearSolver.c:452-481); counts the members that iterate on
__global__ void kb_givens(const ImpDev* __restrict__ I, int m, int* count) {
    MEMBER;
    if (!gmres_on(d)) return;
    const double ww = block_total(d.partial + ((m + 1) & 1) * (d.nb + 1), d.nb);
    if (threadIdx.x) return;
    const int K = d.K;
    double* sc = d.sc;
    double* H = sc + SC_H;  // H[r * (K + 1) + c]
    H[(m + 1) * (K + 1) + m] = sqrt(ww);
    double* gam = H + (K + 1) * (K + 1);
    double* C = gam + (K + 1);
    double* S = C + K;
    double* alp = S + K;
    const int ld = K + 1;
    for (int nn = 0; nn <= m - 1; ++nn) {
        double tmp = C[nn] * H[nn * ld + m] + S[nn] * H[(nn + 1) * ld + m];
        H[(nn + 1) * ld + m] = -S[nn] * H[nn * ld + m] + C[nn] * H[(nn + 1) * ld + m];
        H[nn * ld + m] = tmp;
    }
    double bet = sqrt(H[m * ld + m] * H[m * ld + m] + H[(m + 1) * ld + m] * H[(m + 1) * ld + m]);
    S[m] = H[(m + 1) * ld + m] / bet;
    C[m] = H[m * ld + m] / bet;
    H[m * ld + m] = bet;
    gam[m + 1] = -S[m] * gam[m];
    gam[m] = C[m] * gam[m];
    if ((fabs(gam[m + 1]) <= sc[SC_ABORT]) || (m == K - 1)) {
        for (int nn = m; nn >= 0; --nn) {
            alp[nn] = gam[nn];
            for (int o = nn + 1; o <= m; ++o) alp[nn] -= H[nn * ld + o] * alp[o];
            alp[nn] /= H[nn * ld + nn];
        }
        d.flag[0] = 1;
        d.flag[1] = m;
        if (!isfinite(alp[0])) d.flag[3] = 1;
        d.ctl[CTL_SKIP_GMRES] = 1;
    } else {
        atomicAdd(count, 1);
    }
}

// V[m+1] = W / H[m+1][m] (src/linearSolver.c:496-502)
__global__ void kb_vnext(const ImpDev* __restrict__ I, int m) {
    MEMBER;
    if (!gmres_on(d)) return;
    CELL_INDEX;
    if (i >= d.N) return;
    double w[4];
    ld(d.W[i], w);
    double hh = d.sc[SC_H + (m + 1) * (d.K + 1) + m];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = w[k] / hh;
    putV(d, (long)(m + 1) * d.N + i, mk(w));
}

// end of a GMRES cycle: iteration count, breakdown test
__global__ void kb_gmres_end(const ImpDev* __restrict__ I) {
    MEMBER;
    if (threadIdx.x || !newton_on(d)) return;
    d.ctl[CTL_GMRES_TOTAL] += min(d.flag[1], d.K - 1) + 1;
    if (d.flag[3] || d.flag[4]) fail_member(d, CCFD_ERR_GMRES, FLAG_GMRES);
}

// delX += alp[nn] Z[nn], nn = 0..m in order (src/linearSolver.c:482-490);
// XK += delX, cVar = XK, pVar = consPrim(cVar) (src/timeDiscretization.c:
// 505-520)
__global__ void kb_newton_update(const ImpDev* __restrict__ I) {
    MEMBER;
    if (!newton_on(d)) return;
    CELL_INDEX;
    if (i >= d.N) return;
    const double* alp = d.sc + SC_H + (d.K + 1) * (d.K + 1) + (d.K + 1) + 2 * d.K;
    int m = d.flag[1];
    double x[4];
    ld(d.dX[i], x);
    for (int nn = 0; nn <= m; ++nn) {
        double z[4];
        ld(getZ(d, (long)nn * d.N + i), z);
        double a = alp[nn];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] += a * z[k];
    }
    d.dX[i] = mk(x);
    double xk[4], p[4];
    ld(d.XK[i], xk);
#pragma unroll
    for (int k = 0; k < 4; ++k) xk[k] += x[k];
    double4 xv = mk(xk);
    d.XK[i] = xv;
    d.cons[i] = xv;
    cons_prim(d.gam1, xk, p);
    d.prim[i] = mk(p);
}

// Newton loop test after an update (src/timeDiscretization.c:478-549)
__global__ void kb_newton_check(const ImpDev* __restrict__ I) {
    MEMBER;
    if (threadIdx.x || !newton_on(d)) return;
    int inner = ++d.ctl[CTL_INNER];
    double nk = d.sc[SC_NORM_XK], n0 = d.sc[SC_NORM_X0], eps2loc = d.sc[SC_EPS2LOC];
    if (!isfinite(nk)) {
        fail_member(d, CCFD_ERR_STATE, FLAG_STATE);
        return;
    }
    if ((nk > eps2loc * n0) && (inner < d.n_newton)) return;
    if (inner == d.n_newton) {
        fail_member(d, CCFD_ERR_NEWTON, FLAG_NEWTON);
        return;
    }
    d.ctl[CTL_NEWTON_TOTAL] += inner;
    d.ctl[CTL_NEWTON] = 0;
    d.ctl[CTL_SKIP_NEWTON] = 1;
}

// ---------------------------------------------------------------- Jacobian
// Perturbation of the finite-difference columns.  FP64: sqrt(DBL_EPSILON), as
// buildMatrix (src/linearSolver.c:199).  Mixed precision evaluates the
// columns with FP32 reconstruction and fluxes (the preconditioner only sets
// how fast GMRES converges, not the converged state), where a step below the
// FP32 resolution of the state would vanish: sqrt(FLT_EPSILON), the step that
// balances truncation and rounding error, with an FP32-flux R(U) as base.
__device__ __forceinline__ double jac_eps(const ImpDev& d) {
    return d.fp32 ? sqrt((double)FLT_EPSILON) : sqrt(DBL_EPSILON);
}

// member builds a preconditioner and has colour c
__device__ __forceinline__ bool jac_on(const ImpDev& d, int c) {
    return newton_on(d) && d.precond && c >= 0 && c < d.ncol;
}

// perturbed copies of the state, one per variable (buildMatrix works on a
// copy of pVar)
__global__ void kb_jac_copy(const ImpDev* __restrict__ I) {
    MEMBER;
    if (!newton_on(d) || !d.precond) return;
    CELL_INDEX;
    if (i >= d.N) return;
    const double4 q = d.prim[i];
#pragma unroll
    for (int v = 0; v < 4; ++v) d.pert[v][i] = q;
}

// Between the evaluations of colours c - 1 and c: record the columns of the
// cells of colour c - 1 (the diagonal block of each and the off-diagonal
// blocks of its face neighbours, src/linearSolver.c:203-222), restore their
// states, perturb the cells of colour c and set the skip word of its
// evaluation.  Five threads per cell, the cell itself and its sides; a thread
// has all four columns of its block, so it writes whole block rows.  Bound by
// scattered reads of the columns' residuals: 10 us per colour of a 32,768-cell
// airfoil, where perturbing and recording one variable at a time took four
// evaluations, four recordings and eight perturbations a colour (the implicit
// step 7.5 -> 5.4 ms).
constexpr int kJacParts = 5;

__global__ void __launch_bounds__(128) kb_jac_next(const ImpDev* __restrict__ I, int c) {
    MEMBER;
    const int k = (int)(blockIdx.x * blockDim.x + threadIdx.x) / kJacParts;
    const int part = (int)(blockIdx.x * blockDim.x + threadIdx.x) % kJacParts;
    const bool next = jac_on(d, c);
    if (blockIdx.x == 0 && threadIdx.x == 0) d.ctl[CTL_SKIP_JAC] = !next;
    const double reps = jac_eps(d);
    if (next && part < 4 && k < d.color_off[c + 1] - d.color_off[c]) {
        const int cell = d.color_cells[d.color_off[c] + k];
        double q[4];
        ld(d.prim[cell], q);
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if (v == part) q[v] += reps;
        d.pert[part][cell] = mk(q);
    }
    if (!jac_on(d, c - 1) || k >= d.color_off[c] - d.color_off[c - 1]) return;
    const int cell = d.color_cells[d.color_off[c - 1] + k];
    if (part < 4) d.pert[part][cell] = d.prim[cell];
    // the block this thread records: rows of cell e, columns of `cell`
    int e = cell;
    long t = 16 * (long)cell;
    if (part > 0) {
        const int h = d.hs_off[cell] + part - 1;
        if (h >= d.hs_off[cell + 1]) return;
        e = d.hs_nb[h];
        if (e < 0) return;
        t = 16 * (long)d.twin[h];
    }
    const double sreps = 1.0 / reps, dt = d.ctrl->dt;
    double r[4], u[4][4];
    ld(d.fp32 ? d.rjb[e] : d.RXK[e], r);
#pragma unroll
    for (int v = 0; v < 4; ++v) ld(d.utj[v][e], u[v]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        double o[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) o[v] = 0.0 + (u[v][j] - r[j]) * sreps;
        if (part == 0) {
            *reinterpret_cast<double4*>(d.D + t + 4 * j) = mk(o);
            continue;
        }
        // the off-diagonal blocks of I - dt J (src/linearSolver.c:226-234);
        // the FP32 blocks are rounded before and after the scaling
        if (d.fp32) {
            float f[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) f[v] = (float)((double)(float)o[v] * -dt);
            *reinterpret_cast<float4*>(d.Of + t + 4 * j) = make_float4(f[0], f[1], f[2], f[3]);
        } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) o[v] = o[v] * -dt;
            *reinterpret_cast<double4*>(d.O + t + 4 * j) = mk(o);
        }
    }
}

// own 4x4 inverse by expansion in complementary 2x2 minors; singular when
// |det| <= DBL_EPSILON as in calcDinv
__device__ bool inv4(const double a[16], double r[16]) {
    double s0 = a[0] * a[5] - a[4] * a[1];
    double s1 = a[0] * a[6] - a[4] * a[2];
    double s2 = a[0] * a[7] - a[4] * a[3];
    double s3 = a[1] * a[6] - a[5] * a[2];
    double s4 = a[1] * a[7] - a[5] * a[3];
    double s5 = a[2] * a[7] - a[6] * a[3];
    double c5 = a[10] * a[15] - a[14] * a[11];
    double c4 = a[9] * a[15] - a[13] * a[11];
    double c3 = a[9] * a[14] - a[13] * a[10];
    double c2 = a[8] * a[15] - a[12] * a[11];
    double c1 = a[8] * a[14] - a[12] * a[10];
    double c0 = a[8] * a[13] - a[12] * a[9];
    double det = s0 * c5 - s1 * c4 + s2 * c3 + s3 * c2 - s4 * c1 + s5 * c0;
    if (fabs(det) <= DBL_EPSILON) return false;
    double id = 1.0 / det;
    r[0] = (a[5] * c5 - a[6] * c4 + a[7] * c3) * id;
    r[1] = (-a[1] * c5 + a[2] * c4 - a[3] * c3) * id;
    r[2] = (a[13] * s5 - a[14] * s4 + a[15] * s3) * id;
    r[3] = (-a[9] * s5 + a[10] * s4 - a[11] * s3) * id;
    r[4] = (-a[4] * c5 + a[6] * c2 - a[7] * c1) * id;
    r[5] = (a[0] * c5 - a[2] * c2 + a[3] * c1) * id;
    r[6] = (-a[12] * s5 + a[14] * s2 - a[15] * s1) * id;
    r[7] = (a[8] * s5 - a[10] * s2 + a[11] * s1) * id;
    r[8] = (a[4] * c4 - a[5] * c2 + a[7] * c0) * id;
    r[9] = (-a[0] * c4 + a[1] * c2 - a[3] * c0) * id;
    r[10] = (a[12] * s4 - a[13] * s2 + a[15] * s0) * id;
    r[11] = (-a[8] * s4 + a[9] * s2 - a[11] * s0) * id;
    r[12] = (-a[4] * c3 + a[5] * c1 - a[6] * c0) * id;
    r[13] = (a[0] * c3 - a[1] * c1 + a[2] * c0) * id;
    r[14] = (-a[12] * s3 + a[13] * s1 - a[14] * s0) * id;
    r[15] = (a[8] * s3 - a[9] * s1 + a[10] * s0) * id;
    return true;
}

// I - dt J on the diagonal blocks and their inverses (kb_jac_next has scaled
// the off-diagonal ones: a pass over them took two thirds of this kernel,
// 31 -> 12.5 us on 32,768 cells)
// (src/linearSolver.c:226-251)
__global__ void kb_jac_finish(const ImpDev* __restrict__ I) {
    MEMBER;
    if (!newton_on(d) || !d.precond) return;
    CELL_INDEX;
    if (i >= d.N) return;
    const double dt = d.ctrl->dt;
    double a[16], r[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = d.D[16 * i + k] * -dt;
#pragma unroll
    for (int k = 0; k < 4; ++k) a[5 * k] += 1.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) d.D[16 * i + k] = a[k];
    if (!inv4(a, r)) {
        atomicOr(&d.flag[2], 1);
#pragma unroll
        for (int k = 0; k < 16; ++k) r[k] = 0.0;
    }
    if (d.fp32) {
#pragma unroll
        for (int k = 0; k < 16; ++k) d.Dinvf[16 * i + k] = (float)r[k];
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) d.Dinv[16 * i + k] = r[k];
    }
}

// a singular diagonal block ends the member's step
// (src/linearSolver.c:245-249)
__global__ void kb_jac_check(const ImpDev* __restrict__ I) {
    MEMBER;
    if (threadIdx.x || !newton_on(d) || !d.precond) return;
    if (d.flag[2]) fail_member(d, CCFD_ERR_SINGULAR, FLAG_SINGULAR);
}

// ---------------------------------------------------------------- LU-SGS
// Four consecutive threads treat one cell of a level, thread a its row a:
// forward  dxs_i = Dinv_i (b_i - sum_lower O_ij dxs_j)
// backward dx_i  = dxs_i - Dinv_i (sum_upper O_ij dx_j)
// Row a of the neighbour sum accumulates the neighbours in side order and
// the columns in order, exactly as the reference's loops do; the four rows
// are exchanged by shuffles for the product with Dinv_i.  All loads of a
// cell depend only on its indices (prefetched one level ahead) and on
// results of earlier levels, so they are issued together.
template <typename T> struct Vec4;
template <> struct Vec4<double> { using t = double4; };
template <> struct Vec4<float> { using t = float4; };

template <bool FWD, typename T>
__device__ __forceinline__ void sweep_row(int i, int4 nb, int4 hh, int a, unsigned mask, int lane0,
                                          const T* __restrict__ B, const T* src, T* dst, const T* dxs,
                                          const T* __restrict__ Dinv, const T* __restrict__ O) {
    using V4 = typename Vec4<T>::t;
    const int nbv[4] = {nb.x, nb.y, nb.z, nb.w};
    const int hv[4] = {hh.x, hh.y, hh.z, hh.w};
    // component a of each neighbour state and row a of each block
    T xa[4];
    V4 orow[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (nbv[q] >= 0) {
            xa[q] = src[4 * (long)nbv[q] + a];
            orow[q] = reinterpret_cast<const V4*>(O + 16 * (long)hv[q])[a];
        }
    const V4 drow = reinterpret_cast<const V4*>(Dinv + 16 * (long)i)[a];
    const T own_a = FWD ? B[4 * (long)i + a] : dxs[4 * (long)i + a];
    T t1a = T(0.0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (nbv[q] >= 0) {
            const T o[4] = {orow[q].x, orow[q].y, orow[q].z, orow[q].w};
#pragma unroll
            for (int b = 0; b < 4; ++b) t1a += o[b] * __shfl_sync(mask, xa[q], lane0 + b);
        }
    const T di[4] = {drow.x, drow.y, drow.z, drow.w};
    T t2 = T(0.0);
    if (FWD) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            t2 += di[c] * (__shfl_sync(mask, own_a, lane0 + c) - __shfl_sync(mask, t1a, lane0 + c));
        dst[4 * (long)i + a] = t2;
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) t2 += di[c] * __shfl_sync(mask, t1a, lane0 + c);
        dst[4 * (long)i + a] = own_a - t2;
    }
}

template <bool FWD, typename T>
__device__ __forceinline__ void sweep(int nl, const int* __restrict__ off, const int* __restrict__ cell,
                                      const int4* __restrict__ nbs, const int4* __restrict__ hs,
                                      const T* __restrict__ B, const T* src, T* dst, const T* dxs,
                                      const T* __restrict__ Dinv, const T* __restrict__ O) {
    // the cell count per pass is a multiple of 8, so the four threads of a
    // cell always sit in one aligned quarter of a warp
    const int g = threadIdx.x >> 2, a = threadIdx.x & 3, ng = blockDim.x >> 2;
    const int lane0 = (threadIdx.x & 31) & ~3;
    const unsigned mask = 0xfu << lane0;
    int p = nl > 0 ? off[0] + g : 0;
    int end = nl > 0 ? off[1] : 0;
    bool have = p < end;
    int ci = 0;
    int4 nb = make_int4(-1, -1, -1, -1), hh = nb;
    if (have) {
        ci = cell[p];
        nb = nbs[p];
        hh = hs[p];
    }
    for (int L = 0; L < nl; ++L) {
        // prefetch the first position of the next level
        const int nend = L + 1 < nl ? off[L + 2] : end;
        const int np = end + g;
        const bool nhave = L + 1 < nl && np < nend;
        int nci = 0;
        int4 nnb = make_int4(-1, -1, -1, -1), nhh = nnb;
        if (nhave) {
            nci = cell[np];
            nnb = nbs[np];
            nhh = hs[np];
        }
        if (have) {
            int q = p;
            while (true) {
                sweep_row<FWD, T>(ci, nb, hh, a, mask, lane0, B, src, dst, dxs, Dinv, O);
                q += ng;
                if (q >= end) break;
                ci = cell[q];
                nb = nbs[q];
                hh = hs[q];
            }
        }
        __syncthreads();
        p = np;
        end = nend;
        have = nhave;
        ci = nci;
        nb = nnb;
        hh = nhh;
    }
}

// One CTA per member: the forward sweep, then the backward sweep
// (src/linearSolver.c:261-333): Z_m = LU-SGS(V_m), in the member's precision
// (members of the other precision are left to the other instantiation);
// THREADS / 4 cells of a level per pass.  512 threads: 1024 would take wide
// levels in one pass, but the register cap they impose spills and is slower
// (measured).
template <int THREADS, typename T>
__global__ void __launch_bounds__(THREADS) kb_lusgs(const ImpDev* __restrict__ I, int m) {
    const ImpDev& d = I[blockIdx.x];
    if (!d.precond || !gmres_on(d) || d.fp32 != (sizeof(T) == 4)) return;
    const T *B, *Dinv, *O;
    T *dxs, *dx;
    if constexpr (sizeof(T) == 8) {
        B = reinterpret_cast<const T*>(d.V + (long)m * d.N);
        dxs = reinterpret_cast<T*>(d.dxs);
        dx = reinterpret_cast<T*>(d.Z + (long)m * d.N);
        Dinv = reinterpret_cast<const T*>(d.Dinv);
        O = reinterpret_cast<const T*>(d.O);
    } else {
        B = reinterpret_cast<const T*>(d.Vf + (long)m * d.N);
        dxs = reinterpret_cast<T*>(d.dxsf);
        dx = reinterpret_cast<T*>(d.Zf + (long)m * d.N);
        Dinv = reinterpret_cast<const T*>(d.Dinvf);
        O = reinterpret_cast<const T*>(d.Of);
    }
    sweep<true, T>(d.n_lev_f, d.lev_f_off, d.fw_cell, d.fw_nb, d.fw_h, B, dxs, dxs, dxs, Dinv, O);
    sweep<false, T>(d.n_lev_b, d.lev_b_off, d.bw_cell, d.bw_nb, d.bw_h, B, dx, dx, dxs, Dinv, O);
}

// ---- LU-SGS on a cluster
// One member's sweeps by the warps of a cluster, as a pipeline.  On one SM a
// level costs ~1.5 us: its blocks come through one SM's L2 port, its warps
// share four schedulers, and every level ends in a barrier.  Here each of
// kClWorkers pairs of warps owns a contiguous range of the reference's cell
// numbers and walks its own cells level by level, a chunk of up to eight cells
// (four threads each) at a time.  A cell needs only cells of lower number
// (forward) or higher number (backward), so values flow one way between the
// ranges and the pairs run behind one another without any barrier.  A value
// of the same pair comes from a ring of its recent results; every other value
// is stored by its producer into a mailbox in the consumer's shared memory,
// where the value itself says that it has arrived (mailboxes start as a NaN
// pattern that no result is stored with).  One warp of a pair brings the
// blocks in by cp.async, the other computes: with both in one warp a chunk
// took ~250 instructions of one instruction stream, 1.8 us per level of the
// 32,768-cell airfoil.  The arithmetic and its order are those of sweep_row;
// a missing neighbour is a zero block times a zero vector, which changes no
// sum that starts at +0.  One application on the 32,768-cell airfoil (383 levels
// each way): 0.41 ms (0.53 us per level, a chain of ordered multiply-adds, an
// exchange by shuffles and a mailbox or ring round trip) against 1.18 ms by one
// CTA.
constexpr int kClCtas = 8, kClPairs = 4, kClWorkers = kClCtas * kClPairs, kClThreads = 64 * kClPairs;
constexpr int kClRing = 64;         // recent results of a pair (a power of two)
constexpr int kClMail = 2304;       // mailboxes of a CTA, the first one a zero vector
constexpr int kClNb = 3;            // most neighbours of a cell on one side of the sweep
constexpr int kClSlots = 6;         // chunks whose blocks are in shared memory
constexpr int kClAhead = 3;         // copies in flight, chunks
constexpr int kClIdx = 16;          // chunks whose records are in shared memory
static_assert(kClIdx >= kClSlots + 2 * kClAhead + 1, "a record outlives its blocks");
constexpr int kClSpin = 1 << 25;    // polls (~60 cycles each, about a second) before the sweep gives up

// One place of a chunk: cell (-1: none), half-sides of its blocks in side
// order (-1: none), where the neighbours' values are and where its own result
// goes besides the ring (byte offsets in the CTA's shared memory, the target
// with its CTA in the upper bits, -1: none); neighbours and mailboxes of the
// chunk's busiest place.
struct alignas(16) SweepRec {
    int cell, h[kClNb], src[kClNb], n_nb, mail[4], n_mail, pad[3];  // 64 bytes, copied by four threads
};
constexpr int kClMailBits = 20;
constexpr long kClSpareRecs = 16384;  // records of a sweep: at most four per cell and these

// shared memory of a pair and of a CTA, bytes
template <typename T>
constexpr int cluster_pair_smem() {
    return (int)(kClRing * 4 * sizeof(T) + kClIdx * 8 * sizeof(SweepRec) + kClSlots * 8 * 4 * sizeof(T) +
                 kClSlots * (1 + kClNb) * 32 * 4 * sizeof(T) + 16);
}
template <typename T>
constexpr int cluster_smem() {
    return (int)(kClMail * 4 * sizeof(T)) + kClPairs * cluster_pair_smem<T>();
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(unsigned dst, const void* src, bool take) {
    // without `take` nothing is read and zeros are written
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(take ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ int ld_acquire(unsigned addr) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned addr, int v) {
    asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned map_rank(unsigned addr, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// Values in the ring and the mailboxes: a value whose (upper) word is all ones
// has not arrived; a result of that pattern is stored as the ordinary NaN.
__device__ __forceinline__ double arrivable(double v) {
    return __double2hiint(v) == -1 ? __longlong_as_double(0x7ff8000000000000ll) : v;
}
__device__ __forceinline__ float arrivable(float v) {
    return __float_as_int(v) == -1 ? __int_as_float(0x7fc00000) : v;
}
__device__ __forceinline__ void put_value(unsigned addr, double v) {
    asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void put_value(unsigned addr, float v) {
    asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// the four components at addr; false if one has not arrived
__device__ __forceinline__ bool get_values(unsigned addr, double x[4]) {
    asm volatile("ld.relaxed.cluster.shared::cta.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "r"(addr) : "memory");
    asm volatile("ld.relaxed.cluster.shared::cta.v2.f64 {%0, %1}, [%2];"
                 : "=d"(x[2]), "=d"(x[3])
                 : "r"(addr + 16)
                 : "memory");
    const unsigned a = max((unsigned)__double2hiint(x[0]), (unsigned)__double2hiint(x[1]));
    const unsigned b = max((unsigned)__double2hiint(x[2]), (unsigned)__double2hiint(x[3]));
    return max(a, b) != ~0u;
}
__device__ __forceinline__ bool get_values(unsigned addr, float x[4]) {
    asm volatile("ld.relaxed.cluster.shared::cta.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3])
                 : "r"(addr)
                 : "memory");
    const unsigned a = max(__float_as_uint(x[0]), __float_as_uint(x[1]));
    const unsigned b = max(__float_as_uint(x[2]), __float_as_uint(x[3]));
    return max(a, b) != ~0u;
}

// wait until the other warp's counter at addr is at least `want`; `seen` keeps
// the last value read.  False after kClSpin polls (the whole warp alike).
__device__ __forceinline__ bool reach(unsigned addr, int want, int& seen) {
    for (int n = 0; seen < want; ++n) {
        if (n == kClSpin) return false;
        seen = __shfl_sync(0xffffffffu, ld_acquire(addr), 0);
    }
    return true;
}

// layout of a pair's shared memory from its base
template <typename T>
struct PairSmem {
    unsigned ring, idx, own, rows, full, done;
    __device__ explicit PairSmem(unsigned base) {
        ring = base;                                                    // [kClRing][4]
        idx = ring + (unsigned)(kClRing * 4 * sizeof(T));               // [kClIdx][8] records
        own = idx + (unsigned)(kClIdx * 8 * sizeof(SweepRec));          // [kClSlots][8][4]
        rows = own + (unsigned)(kClSlots * 8 * 4 * sizeof(T));          // [kClSlots][1 + kClNb][units][32] of 16 bytes
        full = rows + (unsigned)(kClSlots * (1 + kClNb) * 32 * 4 * sizeof(T));  // chunks copied
        done = full + 4;                                                // chunks computed
    }
};
template <typename T>
constexpr int kRowUnits = (int)(4 * sizeof(T) / 16);  // 16-byte units of a block row
template <typename T>
constexpr unsigned kSlotBytes = (unsigned)((1 + kClNb) * 32 * 4 * sizeof(T));

// the copying warp of a pair
template <typename T>
__device__ __forceinline__ bool cluster_copy(const PairSmem<T>& S, const int nck, const SweepRec* __restrict__ rec,
                                             const T* own_src, const T* __restrict__ Dinv, const T* __restrict__ O) {
    constexpr int U = kRowUnits<T>;
    const int lane = threadIdx.x & 31, quad = lane >> 2, a = lane & 3;
    auto fetch_idx = [&](int c) {
        if (c < nck)
            cp16(S.idx + (unsigned)((c % kClIdx) * 8 * sizeof(SweepRec)) + 16 * lane,
                 reinterpret_cast<const char*>(rec + 8 * (long)c) + 16 * lane, true);
    };
    for (int c = 0; c < 2 * kClAhead; ++c) fetch_idx(c);
    cp_commit();
    cp_wait<0>();
    __syncwarp();
    int done = 0, slot = 0;
    for (int c = 0; c < nck + kClAhead - 1; ++c) {
        if (c < nck) {
            // the slot's last chunk has been computed
            if (!reach(S.done, c - kClSlots + 1, done)) return false;
            const unsigned r = S.idx + (unsigned)(((c % kClIdx) * 8 + quad) * sizeof(SweepRec));
            int cell, h[kClNb];
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(cell), "=r"(h[0]), "=r"(h[1]), "=r"(h[2])
                         : "r"(r)
                         : "memory");
            const bool have = cell >= 0;
            const long cl = have ? cell : 0;
            const unsigned row = S.rows + slot * kSlotBytes<T> + 16 * lane;
            const char* d = reinterpret_cast<const char*>(Dinv + 16 * cl + 4 * a);
#pragma unroll
            for (int u = 0; u < U; ++u) cp16(row + 512 * u, d + 16 * u, have);
#pragma unroll
            for (int q = 0; q < kClNb; ++q) {
                const char* o = reinterpret_cast<const char*>(O + 16 * (long)max(h[q], 0) + 4 * a);
#pragma unroll
                for (int u = 0; u < U; ++u) cp16(row + 512 * ((q + 1) * U + u), o + 16 * u, h[q] >= 0);
            }
            if (a < U)
                cp16(S.own + (unsigned)((slot * 8 + quad) * 4 * sizeof(T)) + 16 * a,
                     reinterpret_cast<const char*>(own_src + 4 * cl) + 16 * a, have);
            fetch_idx(c + 2 * kClAhead);
            slot = slot + 1 == kClSlots ? 0 : slot + 1;
        }
        cp_commit();
        if (c >= kClAhead - 1) {
            cp_wait<kClAhead - 1>();
            __syncwarp();
            if (lane == 0) st_release(S.full, c - kClAhead + 2);
        }
    }
    return true;
}

// the computing warp of a pair
template <bool FWD, typename T>
__device__ __forceinline__ bool cluster_compute(const PairSmem<T>& S, const unsigned cta, const int nck, T* dst) {
    constexpr int U = kRowUnits<T>;
    const int lane = threadIdx.x & 31, quad = lane >> 2, a = lane & 3, lane0 = lane & ~3;
    int full = 0, slot = 0;
    for (int c = 0; c < nck; ++c) {
        if (!reach(S.full, c + 1, full)) return false;
        __syncwarp();  // also orders the last chunk's results in the ring
        const unsigned rp = S.idx + (unsigned)(((c % kClIdx) * 8 + quad) * sizeof(SweepRec));
        int cell, src[kClNb], n_nb, mail[4], n_mail, skip[3];
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(cell), "=r"(skip[0]), "=r"(skip[1]), "=r"(skip[2])
                     : "r"(rp)
                     : "memory");
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(src[0]), "=r"(src[1]), "=r"(src[2]), "=r"(n_nb)
                     : "r"(rp + 16)
                     : "memory");
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(mail[0]), "=r"(mail[1]), "=r"(mail[2]), "=r"(mail[3])
                     : "r"(rp + 32)
                     : "memory");
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(n_mail) : "r"(rp + 48) : "memory");
        const unsigned row = S.rows + slot * kSlotBytes<T> + 16 * lane;
        auto get_row = [&](int q, T v[4]) {
            if constexpr (sizeof(T) == 8) {
                asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(row + 512 * q * U) : "memory");
                asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                             : "=d"(v[2]), "=d"(v[3])
                             : "r"(row + 512 * (q * U + 1))
                             : "memory");
            } else {
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                             : "r"(row + 512 * q)
                             : "memory");
            }
        };
        T o[kClNb][4], di[4], own_a;
#pragma unroll
        for (int q = 0; q < kClNb; ++q) get_row(q + 1, o[q]);
        get_row(0, di);
        const unsigned oa = S.own + (unsigned)(((slot * 8 + quad) * 4 + a) * sizeof(T));
        if constexpr (sizeof(T) == 8) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(own_a) : "r"(oa) : "memory");
        else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(own_a) : "r"(oa) : "memory");
        T x[kClNb][4];
        for (int n = 0;; ++n) {
            bool here = true;
#pragma unroll
            for (int q = 0; q < kClNb; ++q)
                if (q < n_nb) here = get_values(cta + (unsigned)src[q], x[q]) && here;  // n_nb: the warp's
            if (__all_sync(0xffffffffu, here)) break;
            if (n == kClSpin) return false;
        }
        T t1a = T(0.0);
#pragma unroll
        for (int q = 0; q < kClNb; ++q)
            if (q < n_nb)
#pragma unroll
                for (int b = 0; b < 4; ++b) t1a += o[q][b] * x[q][b];
        const T w = FWD ? own_a - t1a : t1a;
        T t2 = T(0.0);
#pragma unroll
        for (int b = 0; b < 4; ++b) t2 += di[b] * __shfl_sync(0xffffffffu, w, lane0 + b);
        const T res = FWD ? t2 : own_a - t2;
        const T out = arrivable(res);
        put_value(S.ring + (unsigned)((4 * ((8 * c + quad) & (kClRing - 1)) + a) * sizeof(T)), out);
        for (int j = 0; j < n_mail; ++j) {  // the same for the whole warp
            const int to = j == 0 ? mail[0] : j == 1 ? mail[1] : j == 2 ? mail[2] : mail[3];
            if (to >= 0)
                put_value(map_rank(cta + (unsigned)(to & ((1 << kClMailBits) - 1)) + (unsigned)(a * sizeof(T)),
                                   to >> kClMailBits),
                          out);
        }
        if (cell >= 0) __stcg(dst + 4 * (long)cell + a, res);
        slot = slot + 1 == kClSlots ? 0 : slot + 1;
        __syncwarp();
        if (lane == 0) st_release(S.done, c + 1);
    }
    return true;
}

template <typename T>
__global__ void __launch_bounds__(kClThreads) kb_lusgs_cluster(const ImpDev* __restrict__ I, int m) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    grid_wait();
    const ImpDev& d = I[blockIdx.x / kClCtas];
    if (!d.precond || !gmres_on(d) || d.fp32 != (sizeof(T) == 4)) return;  // the whole cluster alike
    const int warp = threadIdx.x >> 5, pair = warp >> 1, w = (blockIdx.x % kClCtas) * kClPairs + pair;
    const unsigned cta = smem_u32(cl_smem);
    const PairSmem<T> S(cta + (unsigned)(kClMail * 4 * sizeof(T)) + pair * cluster_pair_smem<T>());
    const T *B, *Dinv, *O;
    T *dxs, *dx;
    if constexpr (sizeof(T) == 8) {
        B = reinterpret_cast<const T*>(d.V + (long)m * d.N);
        dxs = reinterpret_cast<T*>(d.dxs);
        dx = reinterpret_cast<T*>(d.Z + (long)m * d.N);
        Dinv = reinterpret_cast<const T*>(d.Dinv);
        O = reinterpret_cast<const T*>(d.O);
    } else {
        B = reinterpret_cast<const T*>(d.Vf + (long)m * d.N);
        dxs = reinterpret_cast<T*>(d.dxsf);
        dx = reinterpret_cast<T*>(d.Zf + (long)m * d.N);
        Dinv = reinterpret_cast<const T*>(d.Dinvf);
        O = reinterpret_cast<const T*>(d.Of);
    }
    bool ok = true;
    for (int s = 0; s < 2; ++s) {  // forward, backward
        constexpr int kWords = (int)(kClMail * 4 * sizeof(T) / 16), kZero = kRowUnits<T>;
        for (int k = threadIdx.x; k < kWords; k += kClThreads)
            reinterpret_cast<int4*>(cl_smem)[k] = k < kZero ? make_int4(0, 0, 0, 0) : make_int4(-1, -1, -1, -1);
        if ((threadIdx.x & 63) == 0) {
            st_release(S.full, 0);
            st_release(S.done, 0);
        }
        // every CTA has started, with empty mailboxes; the forward result is
        // complete before the backward sweep requests it
        cluster_sync();
        const int c0 = d.cl_off[s][w], nck = d.cl_off[s][w + 1] - c0;
        const SweepRec* rec = d.cl_rec[s] + 8 * (long)c0;
        bool mine;
        if (warp & 1) mine = cluster_copy<T>(S, nck, rec, s ? dxs : B, Dinv, O);
        else if (s == 0) mine = cluster_compute<true, T>(S, cta, nck, dxs);
        else mine = cluster_compute<false, T>(S, cta, nck, dx);
        ok = ok && mine;
        cp_wait<0>();
        cluster_sync();  // no store into a CTA's memory is still to come
    }
    if (!ok) d.flag[4] = 1;
}

// a vector from / to the reference's cell order (FP32 storage: f)
__global__ void k_vec_in(int n, const double4* __restrict__ src, const int* __restrict__ cell_of_dev,
                         double4* __restrict__ v, float4* __restrict__ f) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    const double4 x = src[cell_of_dev[d]];
    if (f) f[d] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
    else v[d] = x;
}
__global__ void k_vec_out(int n, const double4* __restrict__ v, const float4* __restrict__ f,
                          const int* __restrict__ dev_of_cell, double4* __restrict__ dst) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    if (f) {
        const float4 x = f[dev_of_cell[c]];
        dst[c] = make_double4(x.x, x.y, x.z, x.w);
    } else {
        dst[c] = v[dev_of_cell[c]];
    }
}

// number of members whose Newton loop is still running
__global__ void kb_count(const ImpDev* __restrict__ I, int n, int* out) {
    __shared__ int cnt;
    grid_wait();
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x)
        if (newton_on(I[k])) atomicAdd(&cnt, 1);
    __syncthreads();
    if (threadIdx.x == 0) *out = cnt;
}

}  // namespace

// ------------------------------------------------------------------- host
#define CK(x)                               \
    do {                                    \
        cudaError_t e_ = (x);               \
        if (e_ != cudaSuccess) {            \
            ctx->last_cuda_error = (int)e_; \
            return CCFD_ERR_CUDA;           \
        }                                   \
    } while (0)

template <typename T>
static int ialloc(ccfd_ctx* ctx, T** p, size_t n) {
    void* q = nullptr;
    if (n == 0) n = 1;
    if (ccfd_malloc_async(&q, n * sizeof(T), ctx->stream) != cudaSuccess) return CCFD_ERR_NOMEM;
    ctx->allocs.push_back(q);
    ctx->device_bytes += n * sizeof(T);
    *p = (T*)q;
    return CCFD_OK;
}

template <typename T>
static int iupload(ccfd_ctx* ctx, T** p, const std::vector<T>& h) {
    int st = ialloc(ctx, p, h.size());
    if (st) return st;
    if (!h.empty())
        CK(cudaMemcpyAsync(*p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
    return CCFD_OK;
}

// Host set-up: colouring, twins, level schedules (device cell numbering,
// reference cell order for the sweeps).  Needs the device CSR on the host.
struct ImpSet;
static void set_free(ImpSet* M);

void ccfd_implicit_free(ccfd_ctx* ctx) {
    ImpState* S = (ImpState*)ctx->implicit_state;
    if (S && S->solo) set_free((ImpSet*)S->solo);
    delete S;
    ctx->implicit_state = nullptr;
}

// Records of one cluster sweep: places of the workers' chunks of up to eight
// cells of one level (the same for every cell order on the device); 0 where the
// chunks stay so empty that the sweep is left to the single-CTA kernel.
static long sweep_records(const ccfd_mesh* m, bool fwd) {
    const long N = m->n_cells;
    std::vector<int> lev(N, 0), cnt;
    int nl = 1;
    for (long k = 0; k < N; ++k) {
        const long i = fwd ? k : N - 1 - k;
        int l = 0;
        for (long h = m->hs_offset[i]; h < m->hs_offset[i + 1]; ++h) {
            const long e = m->hs_nb[h];
            if (e >= 0 && (fwd ? e < i : e > i)) l = std::max(l, lev[e] + 1);
        }
        lev[i] = l;
        nl = std::max(nl, l + 1);
    }
    cnt.assign(nl, 0);
    long chunks = 0;
    for (long first = 0, last; first < N; first = last) {
        const long w = first * kClWorkers / N;
        for (last = first; last < N && last * kClWorkers / N == w; ++last) ++cnt[lev[last]];
        for (long i = first; i < last; ++i) {
            chunks += (cnt[lev[i]] + 7) / 8;
            cnt[lev[i]] = 0;
        }
    }
    return 8 * chunks > 4 * N + kClSpareRecs ? 0 : 8 * chunks;
}

// Device bytes of ccfd_implicit_setup, array by array as it allocates them
// (the column scratch by the same first fit into the idle Krylov vectors).
size_t ccfd_implicit_bytes(const ccfd_params* p, const ccfd_mesh* m) {
    const size_t N = m->n_cells, H = m->n_half_sides, F = m->n_faces, B = m->n_bc;
    const size_t K = std::max(1, p->n_kdim), nb = (N + kB - 1) / kB;
    const bool fp32 = p->precision == CCFD_MIXED;
    const size_t vec = fp32 ? sizeof(float4) : sizeof(double4), word = fp32 ? sizeof(float) : sizeof(double);
    size_t b = vec * (2 * K + 1) * N + 8 * sizeof(double4) * N;
    b += sizeof(double) * (SC_H + (K + 1) * (K + 1) + 4 * (K + 1) + 8 + 2 * (nb + 1)) + 4 * (8 + CTL_WORDS);
    if (!p->precond) return b;
    // D, D^-1, off-diagonal blocks, sweep vector, base of the FP32 columns
    b += sizeof(double) * 16 * N + word * 16 * (N + H) + vec * N + (fp32 ? sizeof(double4) * N : 0);
    size_t left[2] = {vec * K * N, vec * K * N};
    auto take = [&](size_t bytes) {
        for (size_t& l : left)
            if (bytes + 256 <= l) {
                l -= bytes + 256;
                return;
            }
        b += bytes;
    };
    for (int v = 0; v < 4; ++v) {
        take(sizeof(double4) * N);
        take(sizeof(double4) * N);
        if (p->spatial_order == 2) take(2 * vec * (p->eqn == CCFD_NAVIER_STOKES ? N : F));
        b += sizeof(double4) * 2 * (B + 1);
    }
    // twins, colours (cells, offsets), levels (cells, neighbours, half-sides,
    // offsets: at most one level per cell), cluster sequences
    b += sizeof(int) * (H + 2 * N) + 2 * (sizeof(int) * 2 + 2 * sizeof(int4)) * N;
    const long fw = sweep_records(m, true), bw = sweep_records(m, false);
    if (fw && bw) b += sizeof(SweepRec) * (fw + bw) + sizeof(int) * 2 * (kClWorkers + 1);
    return b;
}

int ccfd_implicit_setup(ccfd_ctx* ctx, const std::vector<int>& hs_off, const std::vector<int>& hs_nb) {
    ImpState* S = new ImpState();
    ctx->implicit_state = S;
    const long N = ctx->N;
    const int K = std::max(1, ctx->params.n_kdim);
    S->K = K;
    S->N = N;
    S->nb = (int)((N + kB - 1) / kB);
    S->hs_off_h = hs_off;
    const long H = hs_off[N];
    int st;
    S->fp32 = ctx->params.precision == CCFD_MIXED;
    if (S->fp32) {
        if ((st = ialloc(ctx, &S->Vf, (size_t)(K + 1) * N)) || (st = ialloc(ctx, &S->Zf, (size_t)K * N)))
            return st;
    } else if ((st = ialloc(ctx, &S->V, (size_t)(K + 1) * N)) || (st = ialloc(ctx, &S->Z, (size_t)K * N))) {
        return st;
    }
    if ((st = ialloc(ctx, &S->XK, N)) || (st = ialloc(ctx, &S->Q, N)) || (st = ialloc(ctx, &S->RXK, N)) ||
        (st = ialloc(ctx, &S->F, N)) || (st = ialloc(ctx, &S->dX, N)) || (st = ialloc(ctx, &S->W, N)) ||
        (st = ialloc(ctx, &S->ptmp, N)) || (st = ialloc(ctx, &S->ut, N)) ||
        (st = ialloc(ctx, &S->sc, SC_H + (K + 1) * (K + 1) + 4 * (K + 1) + 8)) ||
        (st = ialloc(ctx, &S->flag, 8)) || (st = ialloc(ctx, &S->ctl, CTL_WORDS)) ||
        (st = ialloc(ctx, &S->partial, 2 * ((size_t)S->nb + 1))))
        return st;
    if (ctx->params.precond) {
        if ((st = ialloc(ctx, &S->D, 16 * (size_t)N))) return st;
        if (S->fp32) {
            if ((st = ialloc(ctx, &S->Dinvf, 16 * (size_t)N)) || (st = ialloc(ctx, &S->Of, 16 * (size_t)H)) ||
                (st = ialloc(ctx, &S->RJB, N)) ||
                (st = ialloc(ctx, &S->dxsf, N)))
                return st;
        } else if ((st = ialloc(ctx, &S->Dinv, 16 * (size_t)N)) || (st = ialloc(ctx, &S->O, 16 * (size_t)H)) ||
                   (st = ialloc(ctx, &S->dxs, N))) {
            return st;
        }
        // Scratch of the four columns of a colour.  The Krylov vectors are idle
        // while the Jacobian is built (V_1 .. V_K are written by the
        // iterations after it, Z_0 .. by theirs), so the columns live there
        // as far as they fit.
        {
            const size_t vec = S->fp32 ? sizeof(float4) : sizeof(double4);
            char* at[2] = {S->fp32 ? (char*)(S->Vf + N) : (char*)(S->V + N), S->fp32 ? (char*)S->Zf : (char*)S->Z};
            size_t left[2] = {vec * K * (size_t)N, vec * K * (size_t)N};
            auto take = [&](void** p, size_t bytes) -> int {
                for (int r = 0; r < 2; ++r) {
                    const size_t skip = (size_t)(-(intptr_t)at[r]) & 255;
                    if (skip + bytes <= left[r]) {
                        *p = at[r] + skip;
                        at[r] += skip + bytes;
                        left[r] -= skip + bytes;
                        return CCFD_OK;
                    }
                }
                char* q = nullptr;
                const int e = ialloc(ctx, &q, bytes);
                *p = q;
                return e;
            };
            const bool ns = ctx->params.eqn == CCFD_NAVIER_STOKES;
            const size_t faces = (size_t)(ctx->mesh.F + ctx->mesh.B);
            for (int v = 0; v < 4; ++v)
                if ((st = take((void**)&S->jpert[v], sizeof(double4) * N)) ||
                    (st = take((void**)&S->jut[v], sizeof(double4) * N)) ||
                    (ctx->params.spatial_order == 2 && (st = take(&S->jrec[v], 2 * vec * (ns ? (size_t)N : faces)))) ||
                    (st = ialloc(ctx, &S->jghost[v], 2 * ((size_t)ctx->B + 1))))
                    return st;
        }
        // twins
        std::vector<int> twin(H, -1);
        for (long d = 0; d < N; ++d)
            for (int h = hs_off[d]; h < hs_off[d + 1]; ++h) {
                int e = hs_nb[h];
                if (e < 0) continue;
                for (int g = hs_off[e]; g < hs_off[e + 1]; ++g)
                    if (hs_nb[g] == (int)d) {
                        twin[h] = g;
                        break;
                    }
            }
        // distance-3 colouring: a cell's colour differs from every cell
        // within three face-neighbour steps (greedy in device and in
        // reference order, then colours removed by a bounded tabu search);
        // any valid colouring gives the same entries
        std::vector<int> color;
        const int ncol = ccfd_distance3_colouring(N, hs_off.data(), hs_nb.data(), ctx->dev_of_cell.data(),
                                                  ccfd_colouring_budget(N), color);
        std::vector<int> coff(ncol + 1, 0), ccells(N);
        for (long d = 0; d < N; ++d) coff[color[d] + 1]++;
        for (int c = 0; c < ncol; ++c) coff[c + 1] += coff[c];
        std::vector<int> fill(coff.begin(), coff.end() - 1);
        for (long d = 0; d < N; ++d) ccells[fill[color[d]]++] = (int)d;
        S->color_off = coff;
        // lower / upper neighbour lists in side order, by reference number; a
        // cell that is its own neighbour (a periodic mesh one cell wide) is in
        // neither, as in the reference's loops (src/linearSolver.c:261-333)
        const std::vector<int>& ref = ctx->cell_of_dev;
        std::vector<int> lo_off(N + 1, 0), up_off(N + 1, 0), lo_nb, lo_h, up_nb, up_h;
        for (long d = 0; d < N; ++d) {
            lo_off[d] = (int)lo_nb.size();
            up_off[d] = (int)up_nb.size();
            for (int h = hs_off[d]; h < hs_off[d + 1]; ++h) {
                int e = hs_nb[h];
                if (e < 0 || e == d) continue;
                if (ref[e] < ref[d]) {
                    lo_nb.push_back(e);
                    lo_h.push_back(h);
                } else {
                    up_nb.push_back(e);
                    up_h.push_back(h);
                }
            }
        }
        lo_off[N] = (int)lo_nb.size();
        up_off[N] = (int)up_nb.size();
        // levels, walking the reference numbering
        std::vector<int> lf(N, 0), lb(N, 0);
        const std::vector<int>& dev = ctx->dev_of_cell;
        int nlf = 0, nlb = 0;
        for (long i = 0; i < N; ++i) {
            int d = dev[i], l = 0;
            for (int q = lo_off[d]; q < lo_off[d + 1]; ++q) l = std::max(l, lf[lo_nb[q]] + 1);
            lf[d] = l;
            nlf = std::max(nlf, l + 1);
        }
        for (long i = N - 1; i >= 0; --i) {
            int d = dev[i], l = 0;
            for (int q = up_off[d]; q < up_off[d + 1]; ++q) l = std::max(l, lb[up_nb[q]] + 1);
            lb[d] = l;
            nlb = std::max(nlb, l + 1);
        }
        auto bucket = [&](const std::vector<int>& lev, int nl, std::vector<int>& off, std::vector<int>& cells) {
            off.assign(nl + 1, 0);
            cells.resize(N);
            for (long d = 0; d < N; ++d) off[lev[d] + 1]++;
            for (int l = 0; l < nl; ++l) off[l + 1] += off[l];
            std::vector<int> f(off.begin(), off.end() - 1);
            for (long d = 0; d < N; ++d) cells[f[lev[d]]++] = (int)d;
        };
        std::vector<int> lfo, lfc, lbo, lbc;
        bucket(lf, nlf, lfo, lfc);
        bucket(lb, nlb, lbo, lbc);
        auto pack = [&](const std::vector<int>& cells, const std::vector<int>& off, const std::vector<int>& nb,
                        const std::vector<int>& hh, std::vector<int4>& pn, std::vector<int4>& ph) {
            pn.assign(N, make_int4(-1, -1, -1, -1));
            ph.assign(N, make_int4(-1, -1, -1, -1));
            for (long k = 0; k < N; ++k) {
                int d = cells[k], c = 0;
                int* n4 = &pn[k].x;
                int* h4 = &ph[k].x;
                for (int q = off[d]; q < off[d + 1]; ++q, ++c) {
                    n4[c] = nb[q];
                    h4[c] = hh[q];
                }
            }
        };
        std::vector<int4> fwn, fwh, bwn, bwh;
        pack(lfc, lo_off, lo_nb, lo_h, fwn, fwh);
        pack(lbc, up_off, up_nb, up_h, bwn, bwh);
        // the cluster kernel's sequences; a numbering that needs more
        // mailboxes than a CTA has stays with the single-CTA kernel
        S->cluster_ok = true;
        auto sequences = [&](const std::vector<int>& lev, const std::vector<int>& cells, const std::vector<int4>& pn,
                             const std::vector<int4>& ph, std::vector<int>& off, std::vector<SweepRec>& recs) {
            // cells arrive level by level; each goes to the warp that owns
            // its reference number, into the warp's last chunk if that is of
            // the same level and has room
            std::vector<int> place(N), n_ck(kClWorkers, 0), fill(kClWorkers, 8), last(kClWorkers, -1);
            auto owner = [&](int d) { return (int)((long)ref[d] * kClWorkers / N); };
            for (long k = 0; k < N; ++k) {
                const int d = cells[k], w = owner(d);
                if (fill[w] == 8 || last[w] != lev[d]) {
                    ++n_ck[w];
                    fill[w] = 0;
                    last[w] = lev[d];
                }
                place[d] = 8 * (n_ck[w] - 1) + fill[w]++;
            }
            off.assign(kClWorkers + 1, 0);
            for (int w = 0; w < kClWorkers; ++w) off[w + 1] = off[w] + n_ck[w];
            // (a numbering whose chunks stay nearly empty is left out too:
            // its records would outgrow the memory estimate)
            if (8L * off[kClWorkers] > 4 * N + kClSpareRecs) S->cluster_ok = false;
            if (!S->cluster_ok) return;
            // byte offsets in a CTA's shared memory
            const int word = S->fp32 ? 16 : 32;  // a result
            const int pair_bytes = S->fp32 ? cluster_pair_smem<float>() : cluster_pair_smem<double>();
            SweepRec none;
            memset(&none, 0, sizeof(none));
            none.cell = -1;
            for (int q = 0; q < kClNb; ++q) none.h[q] = -1;  // src 0: the zero vector
            for (int q = 0; q < 4; ++q) none.mail[q] = -1;
            recs.assign(8 * (size_t)off[kClWorkers], none);
            std::vector<int> used(kClCtas, 1);
            for (long k = 0; k < N; ++k) {
                const int d = cells[k], w = owner(d), cta = w / kClPairs;
                SweepRec& r = recs[8 * (size_t)off[w] + place[d]];
                r.cell = d;
                const int *n4 = &pn[k].x, *h4 = &ph[k].x;
                for (int q = 0; q < 4; ++q) {
                    if (n4[q] < 0) continue;
                    if (q >= kClNb) {
                        S->cluster_ok = false;
                        return;
                    }
                    r.h[q] = h4[q];
                    const int e = n4[q], we = owner(e);
                    // the ring holds the last kClRing places before the end
                    // of this chunk
                    if (we == w && place[e] >= (place[d] | 7) + 1 - kClRing) {
                        r.src[q] = word * kClMail + (w % kClPairs) * pair_bytes + word * (place[e] & (kClRing - 1));
                    } else if (used[cta] < kClMail) {
                        const int box = word * used[cta]++;
                        r.src[q] = box;
                        SweepRec& from = recs[8 * (size_t)off[we] + place[e]];
                        int j = 0;
                        while (j < 3 && from.mail[j] >= 0) ++j;  // a cell has at most four neighbours
                        from.mail[j] = (cta << kClMailBits) | box;
                    } else {
                        S->cluster_ok = false;
                        return;
                    }
                }
            }
            for (size_t c = 0; c < recs.size() / 8; ++c) {
                int nn = 0, nm = 0;
                for (int k = 0; k < 8; ++k) {
                    const SweepRec& r = recs[8 * c + k];
                    for (int q = 0; q < kClNb; ++q)
                        if (r.h[q] >= 0) nn = std::max(nn, q + 1);
                    for (int q = 0; q < 4; ++q)
                        if (r.mail[q] >= 0) nm = std::max(nm, q + 1);
                }
                for (int k = 0; k < 8; ++k) {
                    recs[8 * c + k].n_nb = nn;
                    recs[8 * c + k].n_mail = nm;
                }
            }
        };
        std::vector<int> clo[2];
        std::vector<SweepRec> clr[2];
        sequences(lf, lfc, fwn, fwh, clo[0], clr[0]);
        if (S->cluster_ok) sequences(lb, lbc, bwn, bwh, clo[1], clr[1]);
        for (int k = 0; k < 2 && S->cluster_ok; ++k)
            if ((st = iupload(ctx, &S->cl_off[k], clo[k])) || (st = iupload(ctx, &S->cl_rec[k], clr[k]))) return st;
        S->n_lev_f = nlf;
        S->n_lev_b = nlb;
        if ((st = iupload(ctx, &S->twin, twin)) || (st = iupload(ctx, &S->color_cells, ccells)) ||
            (st = iupload(ctx, &S->color_off_d, coff)) ||
            (st = iupload(ctx, &S->lev_f_off, lfo)) || (st = iupload(ctx, &S->fw_cell, lfc)) ||
            (st = iupload(ctx, &S->fw_nb, fwn)) || (st = iupload(ctx, &S->fw_h, fwh)) ||
            (st = iupload(ctx, &S->lev_b_off, lbo)) || (st = iupload(ctx, &S->bw_cell, lbc)) ||
            (st = iupload(ctx, &S->bw_nb, bwn)) || (st = iupload(ctx, &S->bw_h, bwh)))
            return st;
    }
    // a block that no column is recorded in (boundary sides; on a periodic mesh
    // two cells wide the second side of a pair of cells) is zero
    if (S->Of) CK(cudaMemsetAsync(S->Of, 0, sizeof(float) * 16 * (size_t)H, ctx->stream));
    if (S->O) CK(cudaMemsetAsync(S->O, 0, sizeof(double) * 16 * (size_t)H, ctx->stream));
    CK(cudaMemsetAsync(S->sc, 0, sizeof(double) * (SC_H + (K + 1) * (K + 1) + 4 * (K + 1) + 8), ctx->stream));
    CK(cudaMemsetAsync(S->flag, 0, sizeof(int) * 8, ctx->stream));
    CK(cudaMemsetAsync(S->ctl, 0, sizeof(int) * CTL_WORDS, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    S->ready = true;
    return CCFD_OK;
}

// ---------------------------------------------------------------- driver
// A set of implicit members stepped in lockstep on one stream: their device
// descriptors, and per kernel variant the residual-evaluation launch records
// (matrix-vector products at t + dt, Newton residuals at t + dt, Jacobian
// columns at t) over the concatenated tiles of the members.
struct ImpGroup {
    int flux, order, ns, fp32;
    int jac32 = 0;       // Jacobian columns (and their base) with FP32 fluxes (mixed-precision members)
    int n_tiles = 0, smem = 0, smem_jac = 0;
    StageLaunch *rec_mv = nullptr, *rec_nt = nullptr, *rec_jac = nullptr, *rec_jb = nullptr;
    // tile maps of the records: the same tiles with each kind's skip word
    int4 *tmap_mv = nullptr, *tmap_nt = nullptr, *tmap_jac = nullptr, *tmap_jb = nullptr;
};

struct ImpSet {
    std::vector<ccfd_ctx*> members;
    ImpDev* dev = nullptr;
    std::vector<ImpGroup> groups;
    int n = 0, max_nb = 0, max_col = 0, max_colsize = 0, max_K = 0, max_newton = 0;
    bool any_precond = false;
    bool any_plain = false;  // a member without preconditioner
    bool cluster = false;  // LU-SGS by clusters (every preconditioned member fits)
    bool pc64 = false, pc32 = false;  // preconditioned members in FP64 / FP32
    int* d_count = nullptr;
    int* h_count = nullptr;
    int h_count_v = 0;  // ordinary memory: freeing pinned memory would wait for the device
    cudaStream_t stream = nullptr;
    int last_cuda_error = 0;
};

static void set_free(ImpSet* M) {
    if (!M) return;
    for (auto& g : M->groups) {
        cudaFreeAsync(g.rec_mv, M->stream);
        cudaFreeAsync(g.rec_nt, M->stream);
        cudaFreeAsync(g.rec_jac, M->stream);
        cudaFreeAsync(g.rec_jb, M->stream);
        cudaFreeAsync(g.tmap_mv, M->stream);
        cudaFreeAsync(g.tmap_nt, M->stream);
        cudaFreeAsync(g.tmap_jac, M->stream);
        cudaFreeAsync(g.tmap_jb, M->stream);
    }
    if (M->dev) cudaFreeAsync(M->dev, M->stream);
    if (M->d_count) cudaFreeAsync(M->d_count, M->stream);
    delete M;
}

#define CKM(x)                              \
    do {                                    \
        cudaError_t e_ = (x);               \
        if (e_ != cudaSuccess) {            \
            M->last_cuda_error = (int)e_;   \
            return CCFD_ERR_CUDA;           \
        }                                   \
    } while (0)

static ImpDev make_dev(ccfd_ctx* ctx) {
    ImpState* S = (ImpState*)ctx->implicit_state;
    ImpDev d;
    memset(&d, 0, sizeof(d));
    d.N = S->N;
    d.K = S->K;
    d.nb = S->nb;
    d.precond = ctx->params.precond;
    d.n_newton = ctx->params.n_newton_iter;
    d.gam1 = ctx->phys.gam1;
    d.eps_gmres = ctx->params.eps_gmres;
    d.eps2newton = ctx->params.eps_newton * ctx->params.eps_newton;
    d.XK = S->XK; d.Q = S->Q; d.RXK = S->RXK; d.F = S->F; d.dX = S->dX; d.W = S->W;
    d.V = S->V; d.Z = S->Z; d.ptmp = S->ptmp; d.ut = S->ut; d.dxs = S->dxs;
    d.cons = ctx->cons0;
    d.prim = ctx->prim_buf[ctx->cur];
    for (int v = 0; v < 4; ++v) {
        d.pert[v] = S->jpert[v];
        d.utj[v] = S->jut[v];
    }
    d.D = S->D; d.Dinv = S->Dinv; d.O = S->O; d.sc = S->sc; d.partial = S->partial;
    d.fp32 = S->fp32;
    d.Vf = S->Vf; d.Zf = S->Zf; d.dxsf = S->dxsf; d.Dinvf = S->Dinvf; d.Of = S->Of;
    d.rjb = S->RJB;
    d.flag = S->flag;
    d.ctl = S->ctl;
    d.ctrl = ctx->ctrl;
    d.hs_off = ctx->mesh.hs_off;
    d.hs_nb = ctx->mesh.hs_nb;
    d.twin = S->twin;
    d.ncol = ctx->params.precond ? (int)S->color_off.size() - 1 : 0;
    d.color_off = S->color_off_d;
    d.color_cells = S->color_cells;
    d.n_lev_f = S->n_lev_f; d.n_lev_b = S->n_lev_b;
    d.lev_f_off = S->lev_f_off; d.fw_cell = S->fw_cell; d.fw_nb = S->fw_nb; d.fw_h = S->fw_h;
    for (int k = 0; k < 2; ++k) {
        d.cl_off[k] = S->cl_off[k];
        d.cl_rec[k] = S->cl_rec[k];
    }
    d.lev_b_off = S->lev_b_off; d.bw_cell = S->bw_cell; d.bw_nb = S->bw_nb; d.bw_h = S->bw_h;
    return d;
}

// the member's sweeps, if it has any, fit the cluster kernel
static bool sweeps_by_cluster(const ccfd_ctx* ctx) {
    return !ctx->params.precond || ((const ImpState*)ctx->implicit_state)->cluster_ok;
}

static int set_build(const std::vector<ccfd_ctx*>& members, cudaStream_t stream, ImpSet** out) {
    ImpSet* M = new ImpSet();
    *out = M;
    M->members = members;
    M->n = (int)members.size();
    M->stream = stream;
    M->cluster = true;
    for (ccfd_ctx* ctx : members) M->cluster = M->cluster && sweeps_by_cluster(ctx);
    if (M->cluster) {
        CKM(cudaFuncSetAttribute(kb_lusgs_cluster<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 cluster_smem<double>()));
        CKM(cudaFuncSetAttribute(kb_lusgs_cluster<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 cluster_smem<float>()));
    }
    std::vector<ImpDev> hd;
    std::map<std::tuple<int, int, int, int, int>, std::vector<int>> by_variant;
    for (int k = 0; k < M->n; ++k) {
        ccfd_ctx* ctx = members[k];
        ImpState* S = (ImpState*)ctx->implicit_state;
        hd.push_back(make_dev(ctx));
        M->max_nb = std::max(M->max_nb, S->nb);
        M->max_K = std::max(M->max_K, S->K);
        M->max_newton = std::max(M->max_newton, ctx->params.n_newton_iter);
        if (!ctx->params.precond) M->any_plain = true;
        if (ctx->params.precond) {
            M->any_precond = true;
            if (S->fp32) M->pc32 = true;
            else M->pc64 = true;
            int ncol = (int)S->color_off.size() - 1;
            M->max_col = std::max(M->max_col, ncol);
            for (int c = 0; c < ncol; ++c)
                M->max_colsize = std::max(M->max_colsize, S->color_off[c + 1] - S->color_off[c]);
        }
        StageLaunch probe;
        ccfd_fill_stage(ctx, probe);
        by_variant[std::make_tuple(probe.flux_id, probe.order, probe.ns, probe.fp32, (int)S->fp32)].push_back(k);
    }
    CKM(ccfd_malloc_async((void**)&M->dev, sizeof(ImpDev) * M->n, stream));
    CKM(cudaMemcpyAsync(M->dev, hd.data(), sizeof(ImpDev) * M->n, cudaMemcpyHostToDevice, stream));
    CKM(ccfd_malloc_async((void**)&M->d_count, sizeof(int), stream));
    M->h_count = &M->h_count_v;
    for (auto& kv : by_variant) {
        ImpGroup g;
        std::tie(g.flux, g.order, g.ns, g.fp32, g.jac32) = kv.first;
        const std::vector<int>& idx = kv.second;
        std::vector<StageLaunch> mv(idx.size()), nt(idx.size()), jac(4 * idx.size()), jb(idx.size());
        std::vector<int4> tm_mv, tm_nt, tm_jac, tm_jb;
        int max_f = 0;
        for (size_t j = 0; j < idx.size(); ++j) {
            ccfd_ctx* ctx = members[idx[j]];
            ImpState* S = (ImpState*)ctx->implicit_state;
            StageLaunch L;
            ccfd_fill_stage(ctx, L);
            L.ctrl = ctx->ctrl;
            L.mode = 0;
            L.res_partial = ctx->res_partial;
            // matrix-vector product: R(XK + eps Z_m) at t + dt
            L.a_time = 1.0;
            L.prim_in = S->ptmp;
            L.u_t = S->ut;
            L.skip = S->ctl + CTL_SKIP_GMRES;
            mv[j] = L;
            // Newton residual R(XK) at t + dt
            L.prim_in = ctx->prim_buf[ctx->cur];
            L.u_t = S->RXK;
            L.skip = S->ctl + CTL_SKIP_NEWTON;
            nt[j] = L;
            // Jacobian columns at t, one record per variable; they leave the
            // residual partials and the wall pressures of R(XK) alone
            L.a_time = 0.0;
            L.skip = S->ctl + CTL_SKIP_JAC;
            L.fp32 = g.jac32;
            L.res_partial = nullptr;
            L.ghost_pface = nullptr;
            // their base in mixed precision: R(U, t) with FP32 fluxes
            L.u_t = S->RJB;
            jb[j] = L;
            for (int v = 0; v < 4; ++v) {
                L.prim_in = S->jpert[v];
                L.u_t = S->jut[v];
                L.fstate = L.grad = S->jrec[v];
                L.ghosts.state = S->jghost[v];
                L.ghosts.face = S->jghost[v] ? S->jghost[v] + ctx->B + 1 : nullptr;
                jac[4 * j + v] = L;
            }
            for (int t = 0; t < ctx->tiles.n_tiles; ++t) {
                tm_mv.push_back(tile_entry((int)j, t, mv[j].skip));
                tm_nt.push_back(tile_entry((int)j, t, nt[j].skip));
                for (int v = 0; v < 4; ++v) tm_jac.push_back(tile_entry((int)(4 * j + v), t, jac[4 * j].skip));
                tm_jb.push_back(tile_entry((int)j, t, jb[j].skip));
            }
            max_f = std::max(max_f, ctx->tiles.max_f);
        }
        g.n_tiles = (int)tm_mv.size();
        g.smem = stage_smem_bytes(max_f, g.fp32);
        g.smem_jac = stage_smem_bytes(max_f, g.jac32);
        size_t rb = sizeof(StageLaunch) * idx.size();
        CKM(ccfd_malloc_async((void**)&g.rec_mv, rb, stream));
        CKM(ccfd_malloc_async((void**)&g.rec_nt, rb, stream));
        CKM(ccfd_malloc_async((void**)&g.rec_jac, 4 * rb, stream));
        if (g.jac32) {
            CKM(ccfd_malloc_async((void**)&g.rec_jb, rb, stream));
            CKM(cudaMemcpyAsync(g.rec_jb, jb.data(), rb, cudaMemcpyHostToDevice, stream));
        }
        const size_t tb = sizeof(int4) * tm_mv.size();
        CKM(ccfd_malloc_async((void**)&g.tmap_mv, tb, stream));
        CKM(ccfd_malloc_async((void**)&g.tmap_nt, tb, stream));
        CKM(ccfd_malloc_async((void**)&g.tmap_jac, 4 * tb, stream));
        CKM(ccfd_malloc_async((void**)&g.tmap_jb, tb, stream));
        CKM(cudaMemcpyAsync(g.tmap_jb, tm_jb.data(), tb, cudaMemcpyHostToDevice, stream));
        CKM(cudaMemcpyAsync(g.tmap_mv, tm_mv.data(), tb, cudaMemcpyHostToDevice, stream));
        CKM(cudaMemcpyAsync(g.tmap_nt, tm_nt.data(), tb, cudaMemcpyHostToDevice, stream));
        CKM(cudaMemcpyAsync(g.tmap_jac, tm_jac.data(), 4 * tb, cudaMemcpyHostToDevice, stream));
        CKM(cudaMemcpyAsync(g.rec_mv, mv.data(), rb, cudaMemcpyHostToDevice, stream));
        CKM(cudaMemcpyAsync(g.rec_nt, nt.data(), rb, cudaMemcpyHostToDevice, stream));
        CKM(cudaMemcpyAsync(g.rec_jac, jac.data(), 4 * rb, cudaMemcpyHostToDevice, stream));
        M->groups.push_back(g);
    }
    CKM(cudaStreamSynchronize(stream));
    return CCFD_OK;
}

// residual evaluations of a set: matrix-vector products, Newton residuals,
// Jacobian columns, and the FP32-flux base of the columns of mixed-precision
// members (their groups only)
enum RecKind { REC_MV, REC_NT, REC_JAC, REC_JB };

static void residuals(ImpSet* M, RecKind kind) {
    for (auto& g : M->groups) {
        if (kind == REC_JB && !g.jac32) continue;
        const bool jac = kind == REC_JAC || kind == REC_JB;
        BatchLaunch B;
        B.recs = kind == REC_MV ? g.rec_mv : kind == REC_NT ? g.rec_nt : kind == REC_JAC ? g.rec_jac : g.rec_jb;
        B.tmap = kind == REC_MV ? g.tmap_mv : kind == REC_NT ? g.tmap_nt : kind == REC_JAC ? g.tmap_jac : g.tmap_jb;
        B.n_tiles = kind == REC_JAC ? 4 * g.n_tiles : g.n_tiles;
        B.smem_bytes = jac ? g.smem_jac : g.smem;
        B.rk_mode = 0;
        B.stage = 0;
        B.flux_id = g.flux;
        B.order = g.order;
        B.ns = g.ns;
        B.fp32 = jac ? g.jac32 : g.fp32;
        launch_stage_batch(B, M->stream);
    }
}

// buildMatrix + calcDinv (src/linearSolver.c:186-252, :136-179) of the
// members that build a preconditioner: perturbed copies of the state, the
// base of the mixed-precision columns, every colour (its four variables in the
// same launches), blocks and inverses
static void build_jacobian(ImpSet* M, cudaStream_t st) {
    const dim3 gv(M->max_nb, M->n);
    launch_dependent(kb_jac_copy, gv, kB, 0, st, M->dev);
    const dim3 gc((kJacParts * M->max_colsize + 127) / 128, M->n);
    launch_dependent(kb_jac_next, gc, 128, 0, st, M->dev, 0);
    if (M->pc32) residuals(M, REC_JB);
    for (int c = 0; c < M->max_col; ++c) {
        residuals(M, REC_JAC);
        launch_dependent(kb_jac_next, gc, 128, 0, st, M->dev, c + 1);
    }
    launch_dependent(kb_jac_finish, gv, kB, 0, st, M->dev);
}

// LU-SGS of Krylov vector m of every member, a cluster each.  Two implicit
// steps of the first n airfoils of the batched set took, with clusters / one
// CTA per member (ms): n = 16 84 / 180, 32 114 / 196, 64 190 / 273, 128 384 /
// 526; one CTA per member is left to sets with a numbering that needs more
// mailboxes than a CTA has.
template <typename T>
static int launch_lusgs(ImpSet* M, int m, cudaStream_t st) {
    if (!M->cluster) {
        kb_lusgs<kSweepThreads, T><<<M->n, kSweepThreads, 0, st>>>(M->dev, m);
        return CCFD_OK;
    }
    constexpr int smem = cluster_smem<T>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M->n * kClCtas);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    CKM(cudaLaunchKernelEx(&cfg, kb_lusgs_cluster<T>, (const ImpDev*)M->dev, m));
    return CCFD_OK;
}

// members whose Newton loop runs (counted here) / whose GMRES cycle runs
// (counted by the iteration's kb_givens)
static int count_on(ImpSet* M, bool newton, int* out) {
    if (newton) launch_dependent(kb_count, 1, 256, 0, M->stream, M->dev, M->n, M->d_count);
    CKM(cudaMemcpyAsync(M->h_count, M->d_count, sizeof(int), cudaMemcpyDeviceToHost, M->stream));
    CKM(cudaStreamSynchronize(M->stream));
    *out = *M->h_count;
    return CCFD_OK;
}

// One implicitTimeStep (src/timeDiscretization.c:412-552) of every member
// whose control block lets it step, in lockstep.
static int set_step(ImpSet* M) {
    cudaStream_t st = M->stream;
    const dim3 gv(M->max_nb, M->n), g1(1, M->n);
    launch_dependent(kb_step_prepare, g1, 32, 0, st, M->dev);
    launch_dependent(kb_step_begin, gv, kB, 0, st, M->dev);
    residuals(M, REC_NT);
    launch_dependent(kb_newton_F, gv, kB, 0, st, M->dev, 1);
    launch_dependent(kb_newton_norm, g1, kB, 0, st, M->dev, 1);
    launch_dependent(kb_newton_start, g1, 32, 0, st, M->dev);
    CKM(cudaGetLastError());
    for (int it = 0; it < M->max_newton; ++it) {
        int on = 0, s;
        if ((s = count_on(M, true, &on))) return s;
        if (!on) break;
        // GMRES_M (src/linearSolver.c:385-510)
        launch_dependent(kb_gmres_init, gv, kB, 0, st, M->dev);
        launch_dependent(kb_gmres_flags, g1, 32, 0, st, M->dev);
        if (M->any_precond) {
            build_jacobian(M, st);
            launch_dependent(kb_jac_check, g1, 32, 0, st, M->dev);
        }
        for (int m = 0; m < M->max_K; ++m) {
            if (M->pc64 && (s = launch_lusgs<double>(M, m, st))) return s;
            if (M->pc32 && (s = launch_lusgs<float>(M, m, st))) return s;
            if (M->any_plain) launch_dependent(kb_copy_vz, gv, kB, 0, st, M->dev, m);
            // matrixVector: epsFD = sqrt(eps) / |Z|
            launch_dependent(kb_dot_zz, gv, kB, 0, st, M->dev, m, M->d_count);
            const bool sums = M->max_nb > kFusedParts;
            if (sums) launch_dependent(kb_total, g1, kB, 0, st, M->dev, 0);
            launch_dependent(kb_mv_prep, gv, kB, 0, st, M->dev, m);
            residuals(M, REC_MV);
            launch_dependent(kb_mv_finish, gv, kB, 0, st, M->dev, m);
            // modified Gram-Schmidt
            for (int nn = 0; nn <= m; ++nn) {
                if (sums) launch_dependent(kb_total, g1, kB, 0, st, M->dev, nn & 1);
                launch_dependent(kb_mgs, gv, kB, 0, st, M->dev, nn, m);
            }
            launch_dependent(kb_givens, g1, kB, 0, st, M->dev, m, M->d_count);
            launch_dependent(kb_vnext, gv, kB, 0, st, M->dev, m);
            CKM(cudaGetLastError());
            if ((s = count_on(M, false, &on))) return s;
            if (!on) break;
        }
        launch_dependent(kb_gmres_end, g1, 32, 0, st, M->dev);
        launch_dependent(kb_newton_update, gv, kB, 0, st, M->dev);
        residuals(M, REC_NT);
        launch_dependent(kb_newton_F, gv, kB, 0, st, M->dev, 0);
        launch_dependent(kb_newton_norm, g1, kB, 0, st, M->dev, 0);
        launch_dependent(kb_newton_check, g1, 32, 0, st, M->dev);
        CKM(cudaGetLastError());
    }
    // global residual of the final residual evaluation, stop tests and the
    // next dt (calcTimeStep of the new state) of the members that stepped
    for (ccfd_ctx* ctx : M->members)
        imp_step_end_launch(ctx->ctrl, ctx->mesh, ctx->phys, ctx->sp, ctx->res_partial, ctx->tiles.n_tiles,
                            ctx->dt_partial, ctx->dt_bad, ctx->nb_cells, ctx->wall_ghost, ctx->wall_nl,
                            ctx->ghost_pface, ctx->prim_buf[ctx->cur], st);
    CKM(cudaGetLastError());
    return CCFD_OK;
}

// iteration counters of the members into their contexts (reports)
static int set_pull_counts(ImpSet* M) {
    for (ccfd_ctx* ctx : M->members) {
        ImpState* S = (ImpState*)ctx->implicit_state;
        int ctl[CTL_WORDS];
        CKM(cudaMemcpyAsync(ctl, S->ctl, sizeof(ctl), cudaMemcpyDeviceToHost, M->stream));
        CKM(cudaStreamSynchronize(M->stream));
        ctx->newton_total = ctl[CTL_NEWTON_TOTAL];
        ctx->gmres_total = ctl[CTL_GMRES_TOTAL];
    }
    return CCFD_OK;
}

static int run_implicit(ccfd_ctx* ctx, long nsteps, ccfd_report* report) {
    CK(cudaSetDevice(ctx->device));
    ImpState* S = (ImpState*)ctx->implicit_state;
    if (!S || !S->ready) return CCFD_ERR_ARG;
    cudaStream_t st = ctx->stream;
    int s;
    if (!S->solo) {
        ImpSet* M = nullptr;
        s = set_build({ctx}, st, &M);
        S->solo = M;
        if (s) return s;
    }
    ImpSet* M = (ImpSet*)S->solo;
    CK(cudaMemcpyAsync(ctx->h_ctrl, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    Ctrl& c = *ctx->h_ctrl;
    const long long big = (1LL << 62);
    long long stop_at = nsteps > 0 ? c.iter + nsteps : big;
    c.stop_at = stop_at;
    CK(cudaMemcpyAsync(&ctx->ctrl->stop_at, &c.stop_at, sizeof(long long), cudaMemcpyHostToDevice, st));
    CK(cudaEventRecord(ctx->ev_run0, st));
    launch_dt(ctx->mesh, ctx->phys, ctx->ctrl, ctx->sp, ctx->prim_buf[ctx->cur], ctx->dt_partial, ctx->dt_bad, st);
    launch_step_begin(ctx->ctrl, ctx->sp, ctx->dt_partial, ctx->dt_bad, ctx->nb_cells, st);
    CK(cudaMemcpyAsync(ctx->h_ctrl, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    int status = CCFD_OK;
    int ctl_status = 0;
    while (!c.done && c.active && c.iter < stop_at) {
        if ((status = set_step(M))) break;
        CK(cudaMemcpyAsync(ctx->h_ctrl, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&ctl_status, S->ctl + CTL_STATUS, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (ctx->sp.hist && (s = ccfd_history_drain(ctx))) return s;
        if (ctl_status) {
            status = ctl_status;
            break;
        }
    }
    CK(cudaEventRecord(ctx->ev_run1, st));
    CK(cudaEventSynchronize(ctx->ev_run1));
    float run_ms = 0.0f;
    CK(cudaEventElapsedTime(&run_ms, ctx->ev_run0, ctx->ev_run1));
    if ((s = set_pull_counts(M))) return s;
    CK(cudaMemcpyAsync(ctx->h_ctrl, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (report) {
        ccfd_fill_report(ctx, report);
        report->status = status ? status : report->status;
        report->device_ms = run_ms;
    }
    if (status) {
        // a failed step leaves the context usable: clear the stop flags the
        // device raised for it, as the single-case driver always did
        c.done = 0;
        c.active = 0;
        c.flags = 0;
        CK(cudaMemcpyAsync(ctx->ctrl, &c, sizeof(Ctrl), cudaMemcpyHostToDevice, st));
        CK(cudaStreamSynchronize(st));
        return status;
    }
    if (c.flags & FLAG_DT) return CCFD_ERR_DT;
    if (c.flags & FLAG_STATE) return CCFD_ERR_STATE;
    return CCFD_OK;
}

extern "C" int ccfd_run_implicit(ccfd_ctx* ctx, long nsteps, ccfd_report* report) {
    if (!ctx || !ctx->uploaded) return CCFD_ERR_ARG;
    if (ctx->batch) return CCFD_ERR_BUSY;
    return run_implicit(ctx, nsteps, report);
}

// the member set of a context alone (built on first use)
static int solo_set(ccfd_ctx* ctx, ImpSet** out) {
    ImpState* S = (ImpState*)ctx->implicit_state;
    if (!S || !S->ready) return CCFD_ERR_ARG;
    if (!S->solo) {
        ImpSet* M = nullptr;
        int s = set_build({ctx}, ctx->stream, &M);
        S->solo = M;
        if (s) return s;
    }
    *out = (ImpSet*)S->solo;
    return CCFD_OK;
}

// buildMatrix + calcDinv (src/linearSolver.c:136-252) at the context's state
// as at the first Newton iteration of an implicit step from t with time step
// dt, the blocks copied out in the reference's cell and half-side order.
extern "C" int ccfd_build_matrix(ccfd_ctx* ctx, double t, double dt, double* d_out, double* dinv_out,
                                 double* off_out) {
    if (!ctx || !ctx->uploaded || !ctx->params.implicit || !ctx->params.precond) return CCFD_ERR_ARG;
    if (ctx->batch) return CCFD_ERR_BUSY;
    CK(cudaSetDevice(ctx->device));
    ImpSet* M = nullptr;
    int s = solo_set(ctx, &M);
    if (s) return s;
    ImpState* S = (ImpState*)ctx->implicit_state;
    cudaStream_t st = ctx->stream;
    const long N = S->N, H = S->hs_off_h[N];
    // the step's control block (t, dt) and member words (Newton on, no GMRES
    // cycle), restored afterwards
    CK(cudaMemcpyAsync(ctx->h_ctrl, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    const Ctrl saved = *ctx->h_ctrl;
    Ctrl c = saved;
    c.t = t;
    c.dt = dt;
    c.active = 1;
    c.done = 0;
    int ctl[CTL_WORDS] = {0};
    ctl[CTL_NEWTON] = 1;
    ctl[CTL_SKIP_GMRES] = 1;
    CK(cudaMemcpyAsync(ctx->ctrl, &c, sizeof(Ctrl), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(S->ctl, ctl, sizeof(ctl), cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(S->flag, 0, sizeof(int) * 8, st));
    // boundary sides have no block: zero, as the reference's untouched
    // dense entries
    if (S->fp32) CK(cudaMemsetAsync(S->Of, 0, sizeof(float) * 16 * (size_t)H, st));
    else CK(cudaMemsetAsync(S->O, 0, sizeof(double) * 16 * (size_t)H, st));
    const dim3 gv(M->max_nb, M->n), g1(1, M->n);
    residuals(M, REC_NT);  // R_XK = R(U, t + dt)
    build_jacobian(M, st);
    CK(cudaGetLastError());
    std::vector<double> D(16 * N), Di(16 * N), O(16 * H);
    int flag[8];
    CK(cudaMemcpyAsync(D.data(), S->D, sizeof(double) * D.size(), cudaMemcpyDeviceToHost, st));
    if (S->fp32) {
        std::vector<float> a(16 * N), b(16 * H);
        CK(cudaMemcpyAsync(a.data(), S->Dinvf, sizeof(float) * a.size(), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(b.data(), S->Of, sizeof(float) * b.size(), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        for (size_t k = 0; k < a.size(); ++k) Di[k] = a[k];
        for (size_t k = 0; k < b.size(); ++k) O[k] = b[k];
    } else {
        CK(cudaMemcpyAsync(Di.data(), S->Dinv, sizeof(double) * Di.size(), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(O.data(), S->O, sizeof(double) * O.size(), cudaMemcpyDeviceToHost, st));
    }
    CK(cudaMemcpyAsync(flag, S->flag, sizeof(flag), cudaMemcpyDeviceToHost, st));
    int zero[CTL_WORDS] = {0};
    CK(cudaMemcpyAsync(ctx->ctrl, &saved, sizeof(Ctrl), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(S->ctl, zero, sizeof(zero), cudaMemcpyHostToDevice, st));
    CK(cudaStreamSynchronize(st));
    *ctx->h_ctrl = saved;
    S->jac_built = true;
    // device order -> reference order (cells keep their side order)
    long ho = 0;
    for (long cr = 0; cr < N; ++cr) {
        const int d = ctx->dev_of_cell[cr];
        const int h0 = S->hs_off_h[d], nh = S->hs_off_h[d + 1] - h0;
        if (d_out) memcpy(d_out + 16 * cr, &D[16 * (size_t)d], sizeof(double) * 16);
        if (dinv_out) memcpy(dinv_out + 16 * cr, &Di[16 * (size_t)d], sizeof(double) * 16);
        if (off_out) memcpy(off_out + 16 * ho, &O[16 * (size_t)h0], sizeof(double) * 16 * nh);
        ho += nh;
    }
    return flag[2] ? CCFD_ERR_SINGULAR : CCFD_OK;
}

// LUSGS (src/linearSolver.c:261-333) of b with the blocks of the last
// ccfd_build_matrix, in the reference's cell order.
extern "C" int ccfd_lusgs(ccfd_ctx* ctx, const double* b, double* x) {
    if (!ctx || !b || !x || !ctx->uploaded) return CCFD_ERR_ARG;
    if (ctx->batch) return CCFD_ERR_BUSY;
    ImpState* S = (ImpState*)ctx->implicit_state;
    if (!S || !S->jac_built) return CCFD_ERR_ARG;
    CK(cudaSetDevice(ctx->device));
    ImpSet* M = nullptr;
    int s = solo_set(ctx, &M);
    if (s) return s;
    cudaStream_t st = ctx->stream;
    const long N = S->N;
    // b and x pass through the transfer buffer in the reference's order and
    // are permuted (and rounded) on the device
    const unsigned nb = (unsigned)((N + kB - 1) / kB);
    CK(cudaMemcpyAsync(ctx->xfer, b, sizeof(double4) * N, cudaMemcpyHostToDevice, st));
    k_vec_in<<<nb, kB, 0, st>>>((int)N, ctx->xfer, ctx->d_cell_of_dev, S->V, S->Vf);
    CK(cudaMemsetAsync(S->flag + 4, 0, sizeof(int), st));
    CK(cudaMemsetAsync(S->ctl, 0, sizeof(int) * CTL_WORDS, st));  // GMRES "on": the sweep runs
    if ((s = S->fp32 ? launch_lusgs<float>(M, 0, st) : launch_lusgs<double>(M, 0, st))) return s;
    k_vec_out<<<nb, kB, 0, st>>>((int)N, S->Z, S->Zf, ctx->d_dev_of_cell, ctx->xfer);
    CK(cudaGetLastError());
    int gave_up = 0;
    CK(cudaMemcpyAsync(x, ctx->xfer, sizeof(double4) * N, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&gave_up, S->flag + 4, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return gave_up ? CCFD_ERR_GMRES : CCFD_OK;
}

// ---------------------------------------------------------------- batching
// The implicit members of a batch form one lockstep set on the batch stream
// (rebuilt when the membership changes).
// The implicit members of a batch are split into a few lockstep sets, each
// driven by its own host thread on its own stream: the latency-bound work of
// one set (LU-SGS sweeps, reductions) overlaps on the device with the
// throughput-bound residual evaluations of the others.  Rebuilt when the
// membership changes.
struct BatchImp {
    std::vector<ImpSet*> sets;
    std::vector<cudaStream_t> streams;
    std::vector<ccfd_ctx*> key;
};
static std::map<const ccfd_batch*, BatchImp> g_batch_imp;

static void batch_imp_free(BatchImp& bi) {
    for (ImpSet* M : bi.sets) set_free(M);
    for (cudaStream_t st : bi.streams) {
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
    }
    bi.sets.clear();
    bi.streams.clear();
    bi.key.clear();
}

cudaStream_t ccfd_batch_stream(ccfd_batch* b);

int ccfd_implicit_batch_join(ccfd_batch* b, ccfd_ctx* ctx) {
    ImpState* S = (ImpState*)ctx->implicit_state;
    if (!S || !S->ready) return CCFD_ERR_ARG;
    cudaStream_t st = ccfd_batch_stream(b);
    launch_dt(ctx->mesh, ctx->phys, ctx->ctrl, ctx->sp, ctx->prim_buf[ctx->cur], ctx->dt_partial, ctx->dt_bad, st);
    launch_step_begin(ctx->ctrl, ctx->sp, ctx->dt_partial, ctx->dt_bad, ctx->nb_cells, st);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(st));
    return CCFD_OK;
}

int ccfd_implicit_batch_leave(ccfd_batch* b, ccfd_ctx* ctx) {
    auto it = g_batch_imp.find(b);
    if (it != g_batch_imp.end()) {
        for (ImpSet* M : it->second.sets) set_pull_counts(M);
        batch_imp_free(it->second);
        g_batch_imp.erase(it);
    }
    (void)ctx;
    return CCFD_OK;
}

void ccfd_implicit_batch_release(ccfd_batch* b) {
    auto it = g_batch_imp.find(b);
    if (it == g_batch_imp.end()) return;
    batch_imp_free(it->second);
    g_batch_imp.erase(it);
}

// up to `steps` implicit time steps of one lockstep set
static int set_steps(ImpSet* M, int device, int steps) {
    if (cudaSetDevice(device) != cudaSuccess) return CCFD_ERR_CUDA;
    for (int k = 0; k < steps; ++k) {
        // members that can still step
        int any = 0;
        for (ccfd_ctx* ctx : M->members)
            CKM(cudaMemcpyAsync(ctx->h_ctrl, ctx->ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, M->stream));
        CKM(cudaStreamSynchronize(M->stream));
        for (ccfd_ctx* ctx : M->members) any |= ctx->h_ctrl->active && !ctx->h_ctrl->done;
        if (!any) break;
        int s = set_step(M);
        if (s) return s;
    }
    return set_pull_counts(M);
}

int ccfd_implicit_batch_steps(ccfd_batch* b, const std::vector<ccfd_ctx*>& members, int steps) {
    BatchImp& bi = g_batch_imp[b];
    if (bi.key != members) {
        batch_imp_free(bi);
        bi.key = members;
        // sets balanced by cell count (largest first onto the lightest set);
        // at most CCFD_IMPLICIT_SETS (default 8) sets of at least 4 members
        // (256 airfoils: 2 / 4 / 8 / 16 sets 3.17 / 2.93 / 2.75 / 2.87 s;
        // 32 airfoils: 4 and 8 sets alike).  Members whose sweeps need the
        // single-CTA kernel get sets of their own, since a set sweeps by one
        // kernel: eight airfoils, one of them with a shuffled numbering, took
        // 30.0 ms for three steps in one set, 17.0 in two.
        int max_sets = 8;
        if (const char* e = getenv("CCFD_IMPLICIT_SETS")) max_sets = std::max(1, std::min(64, atoi(e)));
        std::vector<int> idx[2];  // by route: any kernel will do or clusters, one CTA
        for (size_t k = 0; k < members.size(); ++k)
            idx[max_sets > 1 && !sweeps_by_cluster(members[k])].push_back((int)k);
        std::vector<std::vector<ccfd_ctx*>> parts;
        int left = max_sets;
        for (int r = 1; r >= 0; --r) {
            if (idx[r].empty()) continue;
            const int most = r && !idx[0].empty() ? left - 1 : left;
            const int n = std::max(1, std::min(most, (int)idx[r].size() / 4));
            left -= n;
            std::stable_sort(idx[r].begin(), idx[r].end(), [&](int a, int c) { return members[a]->N > members[c]->N; });
            const size_t first = parts.size();
            parts.resize(first + n);
            std::vector<long> load(n, 0);
            for (int k : idx[r]) {
                const int j = (int)(std::min_element(load.begin(), load.end()) - load.begin());
                parts[first + j].push_back(members[k]);
                load[j] += members[k]->N;
            }
        }
        const int nsets = (int)parts.size();
        for (int j = 0; j < nsets; ++j) {
            cudaStream_t st;
            if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return CCFD_ERR_CUDA;
            bi.streams.push_back(st);
            ImpSet* M = nullptr;
            int s = set_build(parts[j], st, &M);
            bi.sets.push_back(M);
            if (s) return s;
        }
    }
    int device = members[0]->device;
    std::vector<int> status(bi.sets.size(), CCFD_OK);
    std::vector<std::thread> threads;
    for (size_t j = 1; j < bi.sets.size(); ++j)
        threads.emplace_back([&, j] { status[j] = set_steps(bi.sets[j], device, steps); });
    status[0] = set_steps(bi.sets[0], device, steps);
    for (auto& t : threads) t.join();
    for (int s : status)
        if (s) return s;
    return CCFD_OK;
}
