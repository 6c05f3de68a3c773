// Kernels of the residual-and-update path (templates shared by the
// per-flux translation units stage_fNN.cu, the gradient units gradients*.cu
// and stage.cu).  A residual evaluation or Runge-Kutta stage is two launches:
//
//   k_grad   two threads per cell (second order only): ghost states of its
//            boundary sides at the mirrored barycentres (setBCatBarys,
//            src/boundary.c:320-331), least-squares gradient with
//            Barth-Jespersen / Venkatakrishnan limiting (spatialReconstruction,
//            src/reconstruction.c:198-314), ghost states at the boundary faces
//            (setBCatSides, src/boundary.c:300-314).  Euler: the reconstructed
//            states of the cell's sides go to the face records, so that k_flux
//            streams them; Navier-Stokes: the gradients, which the viscous
//            flux needs as well, and k_flux reconstructs.
//   k_flux   per tile (one CTA): convective and viscous flux of every face of
//            the tile (fluxCalculation, src/fluxCalculation.c:882-998) into
//            shared memory; per-cell sum of the face fluxes in the
//            reference's side order, no atomics (src/finiteVolume.c:96-120);
//            Runge-Kutta stage update with consPrim
//            (src/timeDiscretization.c:362-398); at the last stage the local
//            time step of the new state and the global-residual partial sums;
//            the CTA that finishes last reduces the partials in a fixed order
//            and performs the end-of-step bookkeeping of timeDisc
//            (src/timeDiscretization.c:595-731), the wing coefficients of
//            calcCoef (src/analyze.c:292-387) and the next time step
//   k_dt / k_step_begin   calcTimeStep (src/timeDiscretization.c:249-329)
//            for the first step of a run
//
// Why two launches: a single kernel that staged the tile's states and two
// neighbour rings in shared memory and went through gradients, faces and
// update between barriers took 147 us per stage on the 500,000-triangle
// double Mach reflection (HLLC, Venkatakrishnan, FP64; 108 us with FP32
// fluxes), 344 us on 1,048,576 quads and 28 us on 8,000 quads: at most 24
// warps per SM, ring cells computed twice, half the threads idle in the
// second pass of each phase.  The split keeps each loop's registers low
// enough for 28 warps, computes every gradient once and streams the face
// states: 76, 167 and 13.7 us (62 us with FP32 fluxes), at 0.12 + 0.10 GB of
// DRAM traffic on the 500,000 triangles.  Both kernels are bound by memory
// latency (the scheduler issues in ~42 % of its cycles) and by chains of
// correctly rounded FP64 divisions.
//
// Floating-point operations keep the reference's operand order; the FP64
// units are compiled with -fmad=false, so their results equal the reference's.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "kernels.cuh"

namespace ccfd {

// Dynamic shared memory limit of one kernel, raised as launches need more:
// per device, only ever raised, and safe when host threads (the lockstep
// implicit sets, several serving contexts) launch the same kernel at once.
struct SmemLimit {
    std::mutex mu;
    std::atomic<int> bytes[64];
    SmemLimit() {
        for (auto& b : bytes) b.store(0);
    }
    template <typename K>
    void ensure(K kern, int smem) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
        if (bytes[dev].load(std::memory_order_acquire) >= smem) return;
        std::lock_guard<std::mutex> lk(mu);
        if (bytes[dev].load(std::memory_order_relaxed) >= smem) return;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess)
            bytes[dev].store(smem, std::memory_order_release);
    }
};

// CTA shapes.  k_grad: two threads per cell (kGradVars variables each), at most
// kGradThreads per CTA.
// k_flux: at most `threads`, `single` unless the context sets another size.
// regs / regs_ns (viscous) / grad_regs cap the registers per thread: 76 us per
// stage (500,000 triangles) at 72 registers in k_grad, 84 at 80, 82 at 64 and
// 96; viscous flux 48.9 us (200,000 triangles) at 128, 50.0 at 112, 52.3 at 96.
constexpr int kGradThreads = 128, kGradVars = 2;
template <typename FT> struct StageShape;
template <> struct StageShape<double> { static constexpr int threads = 384, single = 128, regs = 72, regs_ns = 128, grad_regs = 72; };
template <> struct StageShape<float> { static constexpr int threads = 256, single = 128, regs = 64, regs_ns = 72, grad_regs = 64; };

__device__ __forceinline__ double stage_time(const Ctrl* ctrl, double tfix, double a_time) {
    return ctrl ? ctrl->t + a_time * ctrl->dt : tfix;
}

__device__ __forceinline__ bool inactive(const Ctrl* ctrl) { return ctrl && !ctrl->active; }

__device__ __forceinline__ void ld4(const double4& v, double q[4]) {
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
}
__device__ __forceinline__ void ld4(const float4& v, float q[4]) {
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
}
__device__ __forceinline__ double4 mk4(const double q[4]) {
    return make_double4(q[0], q[1], q[2], q[3]);
}
__device__ __forceinline__ float4 mk4(const float q[4]) {
    return make_float4(q[0], q[1], q[2], q[3]);
}

// One 32-byte record per load / store instruction (256-bit accesses; the
// records are 32-byte aligned): a gather then costs one request and one tag
// lookup per sector instead of two.  ld32 is for mesh records, which nothing
// writes while kernels run: to the compiler it is a pure function of the
// address.  What kernels write, this one or the one before it, is loaded by
// ld32_rw and the volatile loads below, which keep their place behind
// grid_wait(), barriers and stores.
__device__ __forceinline__ double4 ld32(const double4* p) {
    double4 v;
    asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
// the same for the viscous flux's face records, which a launch reads once: not
// kept in L1 and first out of L2, so that states and gradients stay there (57.3
// -> 54.5 us per stage on 200,000 triangles; on the half-side and face records
// of the Euler path it gained nothing or, on 1M quads, lost 5 %)
__device__ __forceinline__ double4 ld32_once(const double4* p) {
    double4 v;
    asm("ld.global.L1::no_allocate.L2::evict_first.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
        : "l"(p));
    return v;
}
__device__ __forceinline__ double4 ld32_rw(const double4* p) {
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void st32(double4* p, const double4 v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w)
                 : "memory");
}
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// two consecutive doubles that the kernel may have written itself
__device__ __forceinline__ void ld_rw(const double* p, double (&v)[2]) {
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p) : "memory");
}
// The gradients of a cell are stored variable by variable, (x0, y0, x1, y1),
// (x2, y2, x3, y3), as the threads of the cell write them.
__device__ __forceinline__ void ld_grad(const double4* p, double gx[4], double gy[4]) {
    const double4 a = ld32_rw(p), b = ld32_rw(p + 1);
    gx[0] = a.x; gy[0] = a.y; gx[1] = a.z; gy[1] = a.w;
    gx[2] = b.x; gy[2] = b.y; gx[3] = b.z; gy[3] = b.w;
}
__device__ __forceinline__ void ld_grad(const float4* p, float gx[4], float gy[4]) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(gx[0]), "=f"(gy[0]), "=f"(gx[1]), "=f"(gy[1]), "=f"(gx[2]), "=f"(gy[2]), "=f"(gx[3]), "=f"(gy[3])
                 : "l"(p)
                 : "memory");
}
// the two reconstructed states of a face
__device__ __forceinline__ void ld_face(const double4* p, double l[4], double r[4]) {
    ld4(ld32_rw(p), l);
    ld4(ld32_rw(p + 1), r);
}
__device__ __forceinline__ void ld_face(const float4* p, float l[4], float r[4]) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(l[0]), "=f"(l[1]), "=f"(l[2]), "=f"(l[3]), "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3])
                 : "l"(p)
                 : "memory");
}

// vector types of the stage kernels' arithmetic: FP64 throughout, or FP32
// reconstruction and face fluxes (mixed precision; state, residual sums and
// the update stay FP64)
template <typename T> struct Vec;
template <> struct Vec<double> { using v4 = double4; using v2 = double2; };
template <> struct Vec<float> { using v4 = float4; using v2 = float2; };

template <typename T>
__device__ __forceinline__ typename Vec<T>::v4 cvt4(const double4& v) {
    if constexpr (sizeof(T) == 8) return v;
    else return make_float4(float(v.x), float(v.y), float(v.z), float(v.w));
}
__device__ __forceinline__ double4 to_d4(const double4& v) { return v; }
__device__ __forceinline__ double4 to_d4(const float4& v) {
    return make_double4(v.x, v.y, v.z, v.w);
}

__device__ __forceinline__ double min2(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double max2(double a, double b) { return b > a ? b : a; }
__device__ __forceinline__ float min2(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float max2(float a, float b) { return b > a ? b : a; }

// Limiter value of one side (src/reconstruction.c:25-192): m is the largest
// (u > 0) or smallest (u < 0) neighbour difference, u the reconstructed one.
template <int LIM, typename T>
__device__ __forceinline__ T limiter_value(T m, T u, T eps2) {
    if constexpr (LIM == 1) {
        return m / u;
    } else {
        const T u2 = u * u, m2 = m * m;
        return T(1.0) / u * (((m2 + eps2) * u + T(2.0) * u2 * m) / (m2 + T(2.0) * u2 + u * m + eps2));
    }
}

// Limited least-squares gradient of NV variables of one cell (src/
// reconstruction.c:25-192, 252-312) from their values q, the nh neighbour
// records (nbr(k) points at the variables) and the half-side records (GP.x,
// GP.y, w.x, w.y).  The reference evaluates the limiter of each side with the
// largest or the smallest neighbour difference, by the sign of the
// reconstructed difference; selecting that bound first and evaluating one
// formula keeps warps with both signs from running it twice.  The minimum
// over the sides does not depend on their order.
template <int LIM, int NV, typename T, class Nbr>
__device__ __forceinline__ void cell_gradient(const T q[NV], int nh, T eps2, Nbr nbr,
                                              const double4* __restrict__ gw, T ux[NV], T uy[NV], T gpx[4],
                                              T gpy[4]) {
    T lo[NV], hi[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        lo[v] = hi[v] = q[v];
        ux[v] = uy[v] = T(0.0);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (k < nh) {
            const double4 g = ld32(gw + k);
            double qd[NV];
            ld_rw(nbr(k), qd);
            const T wx = T(g.z), wy = T(g.w);
            gpx[k] = T(g.x);
            gpy[k] = T(g.y);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const T qn = T(qd[v]);
                const T d = qn - q[v];
                ux[v] += wx * d;
                uy[v] += wy * d;
                lo[v] = min2(lo[v], qn);
                hi[v] = max2(hi[v], qn);
            }
        }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const T mn = lo[v] - q[v], mx = hi[v] - q[v];
        T phi = T(1.0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k < nh) {
                const T uD = ux[v] * gpx[k] + uy[v] * gpy[k];
                if (uD > T(0.0) || uD < T(0.0))
                    phi = min2(phi, limiter_value<LIM, T>(uD > T(0.0) ? mx : mn, uD, eps2));
            }
        }
        ux[v] *= phi;
        uy[v] *= phi;
    }
}

// Face flux from the two reconstructed states, rotated into the face frame
// and back, with the viscous contribution, scaled by the face length
// (src/fluxCalculation.c:885-996).  q0 / q1 are the cell-centre states and
// g0x..g1y the cell gradients (Navier-Stokes only).
template <int FLUX, int NS, typename T>
__device__ __forceinline__ void face_flux(const Gas& P, T nx, T ny, T len, const T L[4], const T R[4],
                                          const T q0[4], const T q1[4], const T g0x[4],
                                          const T g0y[4], const T g1x[4], const T g1y[4], double4 bbd,
                                          T F[4], unsigned* flags) {
    // the viscous part first: the gradients and cell states (48 values) are
    // then not live during the convective flux
    T fv[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
    if (NS) {
        T st[4], gx[4], gy[4];
        const T bbz = T(bbd.z);
        T bx = T(bbd.x) / bbz, by = T(bbd.y) / bbz;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            st[v] = T(0.5) * (R[v] + L[v]);
            T gxm = T(0.5) * (g0x[v] + g1x[v]);
            T gym = T(0.5) * (g0y[v] + g1y[v]);
            T corr = gxm * bx + gym * by - (q1[v] - q0[v]) / bbz;
            gx[v] = gxm - corr * bx;
            gy[v] = gym - corr * by;
        }
        T fdx[4], fdy[4];
        diffusion_flux<T>(P, st, gx, gy, fdx, fdy);
#pragma unroll
        for (int v = 0; v < 4; ++v) fv[v] = fdx[v] * nx + fdy[v] * ny;
    }
    FluxIn<T> s;
    s.rL = L[0]; s.uL = nx * L[1] + ny * L[2]; s.vL = -ny * L[1] + nx * L[2]; s.pL = L[3];
    s.rR = R[0]; s.uR = nx * R[1] + ny * R[2]; s.vR = -ny * R[1] + nx * R[2]; s.pR = R[3];
    T fc[4];
    convective_flux<FLUX, T>(P, s, fc, flags);
    F[0] = fc[0];
    F[1] = nx * fc[1] - ny * fc[2];
    F[2] = ny * fc[1] + nx * fc[2];
    F[3] = fc[3];
    if (NS)
#pragma unroll
        for (int v = 0; v < 4; ++v) F[v] -= fv[v];
#pragma unroll
    for (int v = 0; v < 4; ++v) F[v] *= len;
}

// ghost state at the mirrored barycentre of ghost g from interior state q
// (kept out of line: the boundary code is rare and heavy, the hot face code
// should not carry its registers)
static __device__ __noinline__ double4 ghost_bary(const int* __restrict__ gbc, const double4* __restrict__ ggn,
                                           const Phys* __restrict__ Pg, int g, double time, double4 qv,
                                           unsigned* flags) {
    const Phys& P = *Pg;
    double4 gn = ggn[g];
    double x[2] = {gn.x, gn.y};
    double q[4] = {qv.x, qv.y, qv.z, qv.w}, out[4];
    boundary_state(P, P.bc[gbc[g]], gn.z, gn.w, time, q, out, x, flags);
    return make_double4(out[0], out[1], out[2], out[3]);
}

// ghost state at a boundary face from the reconstructed interior face state
static __device__ __noinline__ double4 ghost_face(const int* __restrict__ gbc, const double4* __restrict__ ggn,
                                           const double2* __restrict__ mid, const Phys* __restrict__ Pg,
                                           int g, double time, double4 Lv, unsigned* flags) {
    const Phys& P = *Pg;
    const double4 gn = ggn[g];
    const double2 xm = mid[g];
    double x[2] = {xm.x, xm.y};
    double Lq[4] = {Lv.x, Lv.y, Lv.z, Lv.w}, R[4];
    boundary_state(P, P.bc[gbc[g]], gn.z, gn.w, time, Lq, R, x, flags);
    return make_double4(R[0], R[1], R[2], R[3]);
}

// the same, noting the interior pressure at the face for the wing
// coefficients
__device__ __forceinline__ double4 boundary_face(const StageLaunch& L, int g, double time, double4 q) {
    if (L.ghost_pface) L.ghost_pface[g] = q.w;
    return ghost_face(L.ghosts.bc, L.ghosts.gn, L.ghosts.mid, L.phys_g, g, time, q, L.flags);
}

// owner and neighbour cell (-1-g: ghost g) in a face record's last word
__device__ __forceinline__ int2 face_cells(const double4& nl) {
    return make_int2(__double2loint(nl.w), __double2hiint(nl.w));
}

template <int NV>
__device__ __forceinline__ void block_sum(double v[NV], double* out) {
    __shared__ double sh[NV][32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) sh[k][warp] = v[k];
    __syncthreads();
    if (warp == 0) {
        int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double x = lane < nw ? sh[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) out[k] = x;
        }
    }
}

__device__ __forceinline__ void block_min2(double a, double b, int bad, double2* out, int* bad_out) {
    __shared__ double sa[32], sb[32];
    __shared__ int sbad[32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmin(a, __shfl_down_sync(0xffffffffu, a, o));
        b = fmin(b, __shfl_down_sync(0xffffffffu, b, o));
        bad |= __shfl_down_sync(0xffffffffu, bad, o);
    }
    if (lane == 0) { sa[warp] = a; sb[warp] = b; sbad[warp] = bad; }
    __syncthreads();
    if (warp == 0) {
        int nw = blockDim.x >> 5;
        a = lane < nw ? sa[lane] : 1e150;
        b = lane < nw ? sb[lane] : 1e150;
        bad = lane < nw ? sbad[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = fmin(a, __shfl_down_sync(0xffffffffu, a, o));
            b = fmin(b, __shfl_down_sync(0xffffffffu, b, o));
            bad |= __shfl_down_sync(0xffffffffu, bad, o);
        }
        if (lane == 0) { *out = make_double2(a, b); *bad_out = bad; }
    }
}

// Tile reduction of the last stage: per-thread sums of the four residual
// partials and the minima of the time steps.  The values pass through shared
// memory (red, 6 * blockDim.x doubles) so that one warp finishes one value:
// five shuffle steps per value and CTA instead of per value and warp.
__device__ __forceinline__ void tile_reduce(const double r[4], double dconv, double dvisc, int bad, bool visc,
                                            double* red, double* res_out, double2* dt_out, int* bad_out) {
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;
    __syncthreads();  // red may overlay data other threads still read
#pragma unroll
    for (int v = 0; v < 4; ++v) red[v * nthr + tid] = r[v];
    red[4 * nthr + tid] = dconv;
    if (visc) red[5 * nthr + tid] = dvisc;
    bad = __syncthreads_or(bad);
    for (int v = tid >> 5; v < 6; v += nthr >> 5) {
        double x = v < 4 ? 0.0 : 1e150;
        if (v < 5 || visc)
            for (int i = lane; i < nthr; i += 32) x = v < 4 ? x + red[v * nthr + i] : fmin(x, red[v * nthr + i]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_down_sync(0xffffffffu, x, o);
            x = v < 4 ? x + y : fmin(x, y);
        }
        if (lane == 0) {
            if (v < 4) res_out[v] = x;
            else if (v == 4) dt_out->x = x;
            else dt_out->y = x;
        }
    }
    if (tid == 0) *bad_out = bad;
}

// local convective / viscous time step of one cell (calcTimeStep,
// src/timeDiscretization.c:253-308) at CFL number cfl; returns false if not
// finite
__device__ __forceinline__ bool local_dt(const Gas& P, const StepParams& sp, double cfl, double dfl,
                                         const double q[4], double4 geo, double* dc, double* dv) {
    double a = sqrt(P.gam * q[3] / q[0]);
    *dv = 1e150;
    if (sp.ts1d) {
        *dc = cfl * geo.w / (fabs(q[1]) + a);
        return isfinite(*dc);
    }
    double ssr = (fabs(q[1]) + a) * geo.z + (fabs(q[2]) + a) * geo.w;
    *dc = cfl * geo.x / ssr;
    bool ok = isfinite(*dc);
    if (sp.visc) {
        double ssv = sp.gam_pr_max * P.mu * geo.z * geo.z + sp.gam_pr_max * P.mu * geo.w * geo.w;
        *dv = dfl * q[0] * q[0] * geo.x * geo.x / (4.0 * ssv);
        ok = ok && isfinite(*dv);
    }
    return ok;
}

// global dt from the partial minima with the output / end-time clamp
// (src/timeDiscretization.c:310-321)
__device__ __forceinline__ void finish_dt(Ctrl* ctrl, const StepParams& sp, double dtc, double dtv,
                                          int bad) {
    if (bad) {
        ctrl->flags |= FLAG_DT;
        ctrl->done = 1;
        ctrl->active = 0;
        return;
    }
    double dt = sp.ts1d ? dtc : fmin(dtc, dtv);
    ctrl->visc_dominates = (!sp.ts1d && dtv < dtc) ? 1.0 : 0.0;
    double t = ctrl->t, pT = ctrl->print_time, sT = ctrl->stop_time;
    if ((t + dt > pT) || (t + dt > sT)) dt = fmin(pT, sT) - t;
    else if ((t + 1.5 * dt > pT) || (t + 1.5 * dt > sT)) dt = 0.5 * (fmin(pT, sT) - t);
    ctrl->dt = dt;
}

constexpr int kWallChunk = 256;  // wall faces per pass of the wing-coefficient sums

// End of a step, executed by one whole block: global residual (fixed-order
// reduction of the per-tile partials), wing coefficients, t += dt, the stop
// tests of timeDisc (src/timeDiscretization.c:609-731), the CFL number of
// the next step under switched evolution relaxation and, with with_dt, the
// next dt from the partial minima (otherwise a later k_step_dt computes it
// at the new CFL number).
__device__ __forceinline__ void step_end_block(Ctrl* ctrl, const StepParams& sp, const double* res_partial,
                               int nres, const double2* dt_partial, const int* dt_bad, int ndt,
                               const int* wall_ghost, const double* wall_nl,
                               const double* ghost_pface, const double4* prim_new,
                               bool with_dt = true) {
    __shared__ double s_res[4];
    __shared__ double2 s_dt;
    __shared__ int s_bad;
    const int tid = threadIdx.x;
    double r[4] = {0.0, 0.0, 0.0, 0.0};
    double a = 1e150, b = 1e150;
    int bad = 0;
    // each thread adds its partials in index order; kLd loads are issued at
    // a time, so that the sum over thousands of tiles is not one L2 round
    // trip per partial
    constexpr int kLd = 8;
    const int nthr = blockDim.x;
    for (int i0 = tid; i0 < nres; i0 += kLd * nthr) {
        double2 p[kLd][2];
#pragma unroll
        for (int j = 0; j < kLd; ++j) {
            const int i = i0 + j * nthr;
            const double2* src = reinterpret_cast<const double2*>(res_partial + 4 * (size_t)(i < nres ? i : i0));
            p[j][0] = __ldcg(src);
            p[j][1] = __ldcg(src + 1);
        }
#pragma unroll
        for (int j = 0; j < kLd; ++j)
            if (i0 + j * nthr < nres) {
                r[0] += p[j][0].x;
                r[1] += p[j][0].y;
                r[2] += p[j][1].x;
                r[3] += p[j][1].y;
            }
    }
    for (int i0 = tid; i0 < ndt; i0 += kLd * nthr) {
        double2 p[kLd];
        int e[kLd];
#pragma unroll
        for (int j = 0; j < kLd; ++j) {
            const int i = i0 + j * nthr < ndt ? i0 + j * nthr : i0;
            p[j] = __ldcg(&dt_partial[i]);
            e[j] = __ldcg(&dt_bad[i]);
        }
#pragma unroll
        for (int j = 0; j < kLd; ++j) {
            a = fmin(a, p[j].x);
            b = fmin(b, p[j].y);
            bad |= e[j];
        }
    }
    // wing coefficients: the terms by the whole block, their sums by one
    // thread in the reference's order
    __shared__ double s_wl[2][kWallChunk];
    double cl = 0.0, cd = 0.0;
    if (sp.calc_wing)
        for (int k0 = 0; k0 < sp.n_wall; k0 += kWallChunk) {
            const int n = min(kWallChunk, sp.n_wall - k0);
            for (int k = tid; k < n; k += nthr) {
                const double p0 = __ldcg(&ghost_pface[wall_ghost[k0 + k]]);
                const double* nl = wall_nl + 3 * (size_t)(k0 + k);
                s_wl[0][k] = nl[1] * p0 * nl[2];
                s_wl[1][k] = nl[0] * p0 * nl[2];
            }
            __syncthreads();
            if (tid == 0)
                for (int k = 0; k < n; ++k) {
                    cl += s_wl[0][k];
                    cd += s_wl[1][k];
                }
            __syncthreads();
        }
    block_sum<4>(r, s_res);
    block_min2(a, b, bad, &s_dt, &s_bad);
    __syncthreads();
    if (tid != 0) return;
    double res[6];
#pragma unroll
    for (int v = 0; v < 4; ++v) res[v] = sqrt(s_res[v] * sp.total_area_q);
    res[4] = res[5] = 0.0;
    double dt = ctrl->dt;
    ctrl->t += dt;
    long long iter = ctrl->iter + 1;
    ctrl->iter = iter;
    if (sp.calc_wing) {
        double cl_old = ctrl->cl, cd_old = ctrl->cd;
        cl *= sp.q_inf_lq;
        cd *= sp.q_inf_lq;
        ctrl->cl = cl * sp.cos_a - cd * sp.sin_a;
        ctrl->cd = cd * sp.cos_a + cl * sp.sin_a;
        res[4] = fabs(cl_old - ctrl->cl) / dt;
        res[5] = fabs(cd_old - ctrl->cd) / dt;
    }
#pragma unroll
    for (int v = 0; v < 6; ++v) ctrl->res[v] = res[v];
    if (sp.hist) {
        // the row of this step; the state of other CTAs is read around L1
        double* row = sp.hist + (size_t)((iter - 1) % sp.hist_cap) * sp.hist_width;
        row[0] = (double)iter;
        row[1] = ctrl->t;
        row[2] = dt;
#pragma unroll
        for (int v = 0; v < 6; ++v) row[3 + v] = res[v];
        row[9] = ctrl->cl;
        row[10] = ctrl->cd;
        for (int k = 0; k < sp.n_rec; ++k) {
            const double2* q = reinterpret_cast<const double2*>(&prim_new[sp.rec_cell[k]]);
            double2 a = __ldcg(q), b = __ldcg(q + 1);
            row[kHistHead + 4 * k] = a.x;
            row[kHistHead + 4 * k + 1] = a.y;
            row[kHistHead + 4 * k + 2] = b.x;
            row[kHistHead + 4 * k + 3] = b.y;
        }
    }
    if (!ctrl->have_first) {
#pragma unroll
        for (int v = 0; v < 4; ++v) ctrl->res_first[v] = res[v];
        ctrl->have_first = 1;
    }
    // switched evolution relaxation (Mulder and van Leer, 1985): the CFL
    // number of the next step from the first and the latest residual
    if (sp.ser && res[sp.abort_variable] > 0.0) {
        ctrl->cfl = fmin(sp.ser_cfl_max, sp.cfl * ctrl->res_first[sp.abort_variable] / res[sp.abort_variable]);
        ctrl->dfl = sp.dfl * ctrl->cfl / sp.cfl;
    }
    bool nonfinite = false;
#pragma unroll
    for (int v = 0; v < 4; ++v) nonfinite |= !isfinite(res[v]);
    ctrl->active = 0;
    if (nonfinite) {
        ctrl->flags |= FLAG_STATE;
        ctrl->done = 1;
        return;
    }
    double t = ctrl->t;
    if (ctrl->stop_time - t <= 1e-15) {
        ctrl->finished = 1;
        ctrl->done = 1;
        return;
    }
    if (sp.stationary) {
        double ra = res[sp.abort_variable];
        bool conv = false;
        if (fabs(ra) <= sp.abort_residual) {
            if (sp.abort_on_cl) conv = fabs(res[4]) <= sp.cl_abort;
            else if (sp.abort_on_cd) conv = fabs(res[5]) <= sp.cd_abort;
            else conv = true;
        }
        if (sp.rel_abort > 0.0 && ra <= sp.rel_abort * ctrl->res_first[sp.abort_variable])
            conv = true;
        if (conv) {
            ctrl->converged = 1;
            ctrl->done = 1;
            return;
        }
    }
    if ((ctrl->print_time - t <= 1e-15) || (iter == ctrl->print_iter)) {
        if (ctrl->print_time - t <= 1e-15) ctrl->print_time += ctrl->io_time_interval;
        if (iter == ctrl->print_iter) ctrl->print_iter += ctrl->io_iter_interval;
    }
    if (iter >= ctrl->max_iter) {
        ctrl->max_iter_hit = 1;
        ctrl->done = 1;
        return;
    }
    if (iter >= ctrl->stop_at) return;
    ctrl->active = 1;
    if (with_dt) finish_dt(ctrl, sp, s_dt.x, s_dt.y, s_bad);
}

// limited reconstruction of tile t's cells and the ghost states of their
// boundary sides; two consecutive threads treat one cell, two variables each (a
// fraction of the registers of one thread per cell, so more warps hide the
// gathers).  The boundary code runs in loops of its own over the tile's ghosts,
// before and after the cells: called from the cell loop its registers spilled
// the loop's.
template <int LIM, int NS, typename FT>
__device__ __forceinline__ void grad_body(const StageLaunch& L, const int t) {
    using V4 = typename Vec<FT>::v4;
    constexpr int NV = kGradVars, G = 4 / NV;
    const DevMesh& m = L.mesh;
    const int v0 = NV * (int)(threadIdx.x % G);
    const int d_end = min(m.N, (t + 1) * L.tiles.cells);
    const int2 gr = L.tiles.g_rng[t];
    if (gr.y > 0) {
        const double time = stage_time(L.ctrl, L.tfix, L.a_time);
        for (int i = threadIdx.x; i < gr.y; i += blockDim.x) {
            const int4 e = L.tiles.ghost[gr.x + i];
            L.ghosts.state[e.x] =
                ghost_bary(L.ghosts.bc, L.ghosts.gn, L.phys_g, e.x, time, L.prim_in[e.y], L.flags);
        }
        __syncthreads();
    }
    for (int d = t * L.tiles.cells + (int)(threadIdx.x / G); d < d_end; d += blockDim.x / G) {
        const int4 nb = m.nb4[d];
        const int h0 = m.hs_off[d];
        const int4 sl = NS ? make_int4(0, 0, 0, 0) : m.slot4[d];
        const FT eps2 = LIM == 2 ? FT(m.venk_eps2[d]) : FT(0.0);
        double qd[NV];
        ld_rw(reinterpret_cast<const double*>(L.prim_in + d) + v0, qd);
        const int nbv[4] = {nb.x, nb.y, nb.z, nb.w};
        auto nbr = [&](int k) {
            return reinterpret_cast<const double*>(nbv[k] < 0 ? L.ghosts.state + (-1 - nbv[k]) : L.prim_in + nbv[k]) +
                   v0;
        };
        const int nh = nb.w == kNoSide ? 3 : 4;
        FT q[NV], ux[NV], uy[NV], gpx[4], gpy[4];
#pragma unroll
        for (int v = 0; v < NV; ++v) q[v] = FT(qd[v]);
        cell_gradient<LIM, NV, FT>(q, nh, eps2, nbr, m.hs_gw + h0, ux, uy, gpx, gpy);
        if (NS) {
            FT* g = reinterpret_cast<FT*>(L.grad) + 8 * (size_t)d + 2 * v0;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                g[2 * v] = ux[v];
                g[2 * v + 1] = uy[v];
            }
        }
        if (L.grad_out) {
            double* g = reinterpret_cast<double*>(L.grad_out) + 8 * (size_t)d + 2 * v0;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                g[2 * v] = double(ux[v]);
                g[2 * v + 1] = double(uy[v]);
            }
        }
        // reconstructed states of the sides: Euler into the face records,
        // Navier-Stokes those of boundary sides only
        const int slv[4] = {sl.x, sl.y, sl.z, sl.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k < nh && (!NS || nbv[k] < 0)) {
                FT f[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) f[v] = q[v] + gpx[k] * ux[v] + gpy[k] * uy[v];
                if (NS) {
                    double* o = reinterpret_cast<double*>(L.ghosts.face + (-1 - nbv[k])) + v0;
#pragma unroll
                    for (int v = 0; v < NV; ++v) o[v] = double(f[v]);
                } else {
                    FT* o = reinterpret_cast<FT*>(L.fstate) + 4 * (size_t)slv[k] + v0;
                    *reinterpret_cast<typename Vec<FT>::v2*>(o) = typename Vec<FT>::v2{f[0], f[1]};
                }
            }
        }
    }
    if (gr.y > 0) {
        __syncthreads();
        const double time = stage_time(L.ctrl, L.tfix, L.a_time);
        for (int i = threadIdx.x; i < gr.y; i += blockDim.x) {
            const int4 e = L.tiles.ghost[gr.x + i];
            V4* const fst = reinterpret_cast<V4*>(L.fstate) + e.z;
            const double4 q = NS ? L.ghosts.face[e.x] : to_d4(fst[0]);
            const double4 R = boundary_face(L, e.x, time, q);
            if (NS) L.ghosts.face[e.x] = R;
            else fst[1] = cvt4<FT>(R);
        }
    }
}

// fluxes of the faces of tile t, residual (+ RK stage) of its cells; FT is
// the arithmetic type of the reconstruction and the face fluxes
template <int FLUX, int ORDER, int NS, typename FT>
__device__ __forceinline__ void flux_body(const StageLaunch& L, const int t) {
    using V4 = typename Vec<FT>::v4;
    extern __shared__ double4 smem[];
    using V2 = typename Vec<FT>::v2;
    // face fluxes in two planes of half records: consecutive threads then
    // access consecutive 16 (8) bytes, without bank conflicts
    V2* const fa = reinterpret_cast<V2*>(smem);
    V2* const fb = fa + L.tiles.max_f;
    auto put = [&](int j, const FT q[4]) {
        fa[j] = V2{q[0], q[1]};
        fb[j] = V2{q[2], q[3]};
    };
    auto get = [&](int j, FT q[4]) {
        const V2 a = fa[j], b = fb[j];
        q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y;
    };
    const DevMesh& m = L.mesh;
    const TileDev& T = L.tiles;
    const Gas& P = L.gas;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int4 rng = T.rng[t];
    const int nO = rng.y, nF = rng.y + rng.w;
    const int d0 = t * T.cells, d_end = min(m.N, d0 + T.cells);
    auto face_id = [&](int j) { return j < nO ? rng.x + j : T.border[rng.z + j - nO]; };
    // what the update of this thread's first cell will read
    if (d0 + tid < d_end) {
        prefetch_l1(T.u_code + d0 + tid);
        prefetch_l1(m.area_q + d0 + tid);
        if (L.mode == 1) prefetch_l1(L.cons0 + d0 + tid);
    }

    // source term of the tile's cells (calcSource), evaluated first, while
    // few registers are live, into a per-cell buffer that the same thread
    // reads back below (same cell-to-thread mapping)
    if (m.cell_src) {
        const double time = stage_time(L.ctrl, L.tfix, L.a_time);
        for (int d = d0 + tid; d < d_end; d += nthr)
            m.src_buf[d] = cell_source(*L.phys_g, m.hs_gw, m.hs_off[d], m.hs_off[d + 1], m.cell_src[d],
                                       m.cell_geo[d].x, time);
    }

    if (ORDER == 1) {
        // first order: the ghost states of the boundary faces, from the cell
        // states (in second order k_grad has written them)
        const int2 gr = T.g_rng[t];
        if (gr.y > 0) {
            const double time = stage_time(L.ctrl, L.tfix, L.a_time);
            for (int i = tid; i < gr.y; i += nthr) {
                const int4 e = T.ghost[gr.x + i];
                L.ghosts.face[e.x] = boundary_face(L, e.x, time, to_d4(cvt4<FT>(L.prim_in[e.y])));
            }
            __syncthreads();
        }
    }

    // fluxes of the tile's faces
    int id_next = tid < nF ? face_id(tid) : 0;
    for (int j = tid; j < nF; j += nthr) {
        const int id = id_next;
        if (j + nthr < nF) id_next = face_id(j + nthr);
        const double4 nl = ld32(T.f_nl + id);
        FT q0[4] = {0, 0, 0, 0}, q1[4] = {0, 0, 0, 0}, Lf[4], Rf[4];
        FT g0x[4] = {0, 0, 0, 0}, g0y[4] = {0, 0, 0, 0}, g1x[4] = {0, 0, 0, 0}, g1y[4] = {0, 0, 0, 0};
        double4 bb = make_double4(0, 0, 1, 0);
        if (ORDER == 2 && !NS) {
            ld_face(reinterpret_cast<const V4*>(L.fstate) + 2 * (size_t)id, Lf, Rf);
        } else {
            // ghost cells: a state at the mirrored barycentre in second
            // order (zero in first order, as in the reference), no gradient
            const int2 lr = face_cells(nl);
            const bool inner = lr.y >= 0;
            if (NS) bb = ld32_once(T.f_bb + id);
            ld4(cvt4<FT>(ld32_rw(L.prim_in + lr.x)), q0);
            if (inner) ld4(cvt4<FT>(ld32_rw(L.prim_in + lr.y)), q1);
            else if (ORDER == 2) ld4(cvt4<FT>(ld32_rw(L.ghosts.state + (-1 - lr.y))), q1);
            if (ORDER == 2) {
                const V4* grad = reinterpret_cast<const V4*>(L.grad);
                const double4 gp = ld32_once(T.f_gp + id);
                const FT pxl = FT(gp.x), pyl = FT(gp.y), pxr = FT(gp.z), pyr = FT(gp.w);
                ld_grad(grad + 2 * (size_t)lr.x, g0x, g0y);
#pragma unroll
                for (int v = 0; v < 4; ++v) Lf[v] = q0[v] + pxl * g0x[v] + pyl * g0y[v];
                if (inner) {
                    ld_grad(grad + 2 * (size_t)lr.y, g1x, g1y);
#pragma unroll
                    for (int v = 0; v < 4; ++v) Rf[v] = q1[v] + pxr * g1x[v] + pyr * g1y[v];
                }
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    Lf[v] = q0[v];
                    Rf[v] = q1[v];
                }
            }
            if (!inner) ld4(cvt4<FT>(ld32_rw(L.ghosts.face + (-1 - lr.y))), Rf);
        }
        FT F[4];
        face_flux<FLUX, NS, FT>(P, FT(nl.x), FT(nl.y), FT(nl.z), Lf, Rf, q0, q1, g0x, g0y, g1x, g1y, bb, F, L.flags);
        put(j, F);
    }
    __syncthreads();

    // per-cell flux sum in side order, update
    double r[4] = {0, 0, 0, 0};
    double dconv = 1e150, dvisc = 1e150;
    int bad = 0;
    const bool rk = L.mode == 1;
    for (int d = d0 + tid; d < d_end; d += nthr) {
        const ushort4 code = T.u_code[d];
        const unsigned cv[4] = {code.x, code.y, code.z, code.w};
        double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (cv[k] != 0xffffu) {
                FT F[4];
                get(cv[k] >> 1, F);
                const bool neg = cv[k] & 1u;
#pragma unroll
                for (int v = 0; v < 4; ++v) s[v] += neg ? -double(F[v]) : double(F[v]);
            }
        }
        const double4 sv = m.cell_src ? m.src_buf[d] : make_double4(0.0, 0.0, 0.0, 0.0);
        const double src[4] = {sv.x, sv.y, sv.z, sv.w};
        const double aq = m.area_q[d];
        double ut[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) ut[v] = (src[v] - s[v]) * aq;
        if (L.u_t) st32(L.u_t + d, mk4(ut));
        if (rk) {
            double c0[4], cn[4], pn[4];
            ld4(ld32_rw(L.cons0 + d), c0);
            double adt = L.rk * L.ctrl->dt;
#pragma unroll
            for (int v = 0; v < 4; ++v) cn[v] = c0[v] + adt * ut[v];
            cons_prim(P.gam1, cn, pn);
            st32(L.prim_out + d, mk4(pn));
            if (L.last_stage) {
                st32(L.cons0 + d, mk4(cn));
                double a, b;
                if (!local_dt(P, L.sp, L.sp.cfl, L.sp.dfl, pn, m.cell_geo[d], &a, &b)) bad = 1;
                else {
                    dconv = fmin(dconv, a);
                    dvisc = fmin(dvisc, b);
                }
            }
        }
        if (L.res_partial) {
            const double area = m.cell_geo[d].x;
#pragma unroll
            for (int v = 0; v < 4; ++v) r[v] += area * ut[v] * ut[v];
        }
    }
    if (L.dt_partial) {
        tile_reduce(r, dconv, dvisc, bad, L.sp.visc, reinterpret_cast<double*>(smem), &L.res_partial[4 * t],
                    &L.dt_partial[t], &L.dt_bad[t]);
    } else if (L.res_partial) {
        double out[4];
        block_sum<4>(r, out);
        if (tid == 0)
#pragma unroll
            for (int v = 0; v < 4; ++v) L.res_partial[4 * t + v] = out[v];
    }
    if (rk && L.last_stage) {
        // the CTA that finishes last closes the step (one thread's fence
        // covers what the CTA wrote before the barrier)
        __shared__ int s_last;
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            s_last = atomicAdd(L.ticket, 1u) == (unsigned)(T.n_tiles - 1);
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            Ctrl* ctrl = const_cast<Ctrl*>(L.ctrl);
            step_end_block(ctrl, L.sp, L.res_partial, T.n_tiles, L.dt_partial, L.dt_bad, T.n_tiles,
                           L.wall_ghost, L.wall_nl, L.ghost_pface, L.prim_out);
            if (tid == 0) {
                ctrl->par ^= (L.sp.nrk & 1);  // buffer holding the state after this step
                *L.ticket = 0u;
            }
        }
    }
}

// one instance: one tile per CTA, launch parameters in the parameter space
template <int LIM, int NS, typename FT>
__global__ void __maxnreg__(StageShape<FT>::grad_regs) k_grad(const __grid_constant__ StageLaunch L) {
    grid_wait();
    if (inactive(L.ctrl)) return;
    grad_body<LIM, NS, FT>(L, blockIdx.x);
}

template <int FLUX, int ORDER, int NS, typename FT>
__global__ void __maxnreg__(NS ? StageShape<FT>::regs_ns : StageShape<FT>::regs) k_flux(const __grid_constant__ StageLaunch L) {
    grid_wait();
    if (inactive(L.ctrl)) return;
    // last tile first: what k_grad wrote last is still in L2, and the next
    // k_grad starts with the states written last here
    flux_body<FLUX, ORDER, NS, FT>(L, L.tiles.n_tiles - 1 - (int)blockIdx.x);
}

// Many instances in one launch over their concatenated tiles: entry b of the
// tile map names the instance, its tile and the word that says whether the
// instance steps.  The CTA copies the instance's record to shared memory
// while one thread reads that word (one round trip after the map entry); an
// RK stage then takes its state buffers from the parity in the control block
// and its coefficients from the instance's table.  False: nothing to do.
__device__ __forceinline__ bool batch_record(const StageLaunch* __restrict__ recs, const int4 e, int rk_mode,
                                             int stage, StageLaunch& L) {
    static_assert(sizeof(StageLaunch) % 16 == 0, "launch record copied in 16-byte words");
    constexpr int W = (int)(sizeof(StageLaunch) / 16);
    __shared__ int s_go, s_par;
    const int4* src = reinterpret_cast<const int4*>(recs + e.x);
    for (int k = threadIdx.x; k < W; k += blockDim.x) reinterpret_cast<int4*>(&L)[k] = src[k];
    if (threadIdx.x == 0) {
        const unsigned long long w = ((unsigned long long)(unsigned)e.w << 32) | (unsigned)e.z;
        if (rk_mode) {
            const Ctrl* cb = reinterpret_cast<const Ctrl*>(w);
            s_go = cb->active;
            s_par = cb->par;
        } else {
            const int* skip = reinterpret_cast<const int*>(w);
            s_go = !(skip && *skip);
        }
    }
    __syncthreads();
    if (!s_go) return false;
    if (rk_mode) {
        if (stage >= L.sp.nrk) return false;
        __syncthreads();  // every thread has read nrk and the go word
        if (threadIdx.x == 0) {
            const int in = s_par ^ (stage & 1);
            L.prim_in = L.prim_buf[in];
            L.prim_out = L.prim_buf[in ^ 1];
            L.a_time = L.sp.rk[stage];
            L.rk = L.sp.rk[stage + 1];
            L.last_stage = stage == L.sp.nrk - 1;
            if (!L.last_stage) {
                L.res_partial = nullptr;
                L.dt_partial = nullptr;
            }
        }
        __syncthreads();
    }
    return true;
}

template <int NS, typename FT>
__global__ void __maxnreg__(StageShape<FT>::grad_regs)
    k_grad_batch(const StageLaunch* __restrict__ recs, const int4* __restrict__ tmap, int rk_mode, int stage) {
    __shared__ __align__(16) unsigned char rec[sizeof(StageLaunch)];
    StageLaunch& L = *reinterpret_cast<StageLaunch*>(rec);
    const int4 e = tmap[blockIdx.x];
    grid_wait();
    if (!batch_record(recs, e, rk_mode, stage, L)) return;
    if (L.limiter == 1) grad_body<1, NS, FT>(L, e.y);
    else grad_body<2, NS, FT>(L, e.y);
}

template <int FLUX, int ORDER, int NS, typename FT>
__global__ void __maxnreg__(NS ? StageShape<FT>::regs_ns : StageShape<FT>::regs)
    k_flux_batch(const StageLaunch* __restrict__ recs, const int4* __restrict__ tmap, int rk_mode, int stage) {
    __shared__ __align__(16) unsigned char rec[sizeof(StageLaunch)];
    StageLaunch& L = *reinterpret_cast<StageLaunch*>(rec);
    const int4 e = tmap[gridDim.x - 1 - blockIdx.x];
    grid_wait();
    if (!batch_record(recs, e, rk_mode, stage, L)) return;
    flux_body<FLUX, ORDER, NS, FT>(L, e.y);
}

// dynamic shared memory of a k_flux CTA: the tile's face fluxes, overlaid by
// the last stage's reduction
template <typename FT>
inline int stage_smem_bytes_t(int max_f, int threads) {
    const int flux = (int)sizeof(typename Vec<FT>::v4) * max_f, red = (int)sizeof(double) * 6 * threads;
    return flux > red ? flux : red;
}

// gradient kernels (gradients.cu, gradients_mixed.cu)
void launch_grad_fp64(const StageLaunch& L, cudaStream_t st);
void launch_grad_fp32(const StageLaunch& L, cudaStream_t st);
void launch_grad_batch_fp64(const BatchLaunch& B, cudaStream_t st);
void launch_grad_batch_fp32(const BatchLaunch& B, cudaStream_t st);

// per-flux entry points (stage_fNN.cu)
#define CCFD_DECLARE_FLUX(ID)                                             \
    void launch_stage_f##ID(const StageLaunch& L, cudaStream_t st);       \
    void launch_stage_batch_f##ID(const BatchLaunch& B, cudaStream_t st);
CCFD_DECLARE_FLUX(1) CCFD_DECLARE_FLUX(2) CCFD_DECLARE_FLUX(3) CCFD_DECLARE_FLUX(4)
CCFD_DECLARE_FLUX(5) CCFD_DECLARE_FLUX(6) CCFD_DECLARE_FLUX(7) CCFD_DECLARE_FLUX(8)
CCFD_DECLARE_FLUX(9) CCFD_DECLARE_FLUX(10) CCFD_DECLARE_FLUX(11)
#undef CCFD_DECLARE_FLUX

}  // namespace ccfd
