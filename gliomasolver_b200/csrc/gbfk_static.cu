// gbfk_rd_step_static: one fused RD step on a uniform periodic grid that
// allocates no device memory.
//
// Who needs it: a caller whose device memory is owned by another allocator
// (a framework that reserved the GPU's memory up front and hands out
// sub-buffers), or a time loop that must not pay cudaMalloc's device-wide
// synchronisation, cannot let the library allocate its per-call scratch.
// This variant has none: one kernel reads the caller's p_w, p_g and phi and
// writes the next phi, and everything between them lives in shared memory.
//
// Limits:
//  - at most GBFK_STATIC_MAX_BLOCKS (512) blocks of 8^3 cells, i.e. up to a
//    64^3 grid; larger grids are rejected with GBFK_E_TOO_LARGE.  A larger
//    grid's loop should keep its face coefficients between steps, as
//    gbfk_rd_step does;
//  - no NaN check: a step that produces NaN or Inf returns GBFK_OK;
//  - the caller's current device is restored before returning; an error that
//    the caller's earlier work left pending is returned as GBFK_E_CUDA and
//    not cleared.
// Calls share nothing, so they may overlap on the GPU as far as their own
// buffers allow.
#include "gbfk.h"
#include "gbfk_exact.cuh"
#include "gbfk_kernels.cuh"

#include <cuda_runtime.h>

#include <cstdint>

namespace gbfk {
namespace {

// A block's cells and its six face halos: phi, df = p_w*Dw + p_g*Dg and the
// no-flux test, each formed once per cell of the lab.
template <typename Real>
struct StaticLab {
    Real phi[kLab3], df[kLab3];
    unsigned char low[kLab3];
};

__device__ __forceinline__ int lab_at(int x, int y, int z) { return (x + 1) + kLab * ((y + 1) + kLab * (z + 1)); }

// One CTA per 8^3 block (block b = bx + bpd*(by + bpd*bz), cell x fastest).
//
// What bounds it is the chain of one call, not bandwidth: the largest grid's
// four fields are 4 MB (FP32).  So a step is one launch with two dependent
// stages, load and compute.  Before, it was a topology kernel, a memset, the
// face coefficients through global memory (7.3 MiB of scratch) and the step.
// A face's harmonic mean is formed by both of its cells: its value is the same
// from either side, the division's latency is hidden by the other faces, and
// one more barrier and 1728 words of shared memory would cost more.  One cell
// per thread: 4.7 us at 32^3 (FP32) against 5.8 with two cells per thread,
// 5.5 against 6.9 at 64^3.  A call from Python went from 18.2 to 12.0 us at
// every size, what is left is the caller's and the launch.
template <typename Real>
__global__ void __launch_bounds__(kBS3, 2)
static_step_kernel(int bpd, const Real *__restrict__ pw, const Real *__restrict__ pg, const Real *__restrict__ phi_in,
                   Real *__restrict__ phi_out, Real Dw, Real Dg, Real rho, double ih2, double dt)
{
    __shared__ StaticLab<Real> S;
    const int t = threadIdx.x, b = blockIdx.x;
    const int bx = b % bpd, by = (b / bpd) % bpd, bz = b / (bpd * bpd);
    const int64_t base = (int64_t)b * kBS3;
    auto put = [&](int l, int64_t g) -> bool {
        const Real w = pw[g], q = pg[g], p = phi_in[g];
        S.phi[l] = p;
        S.df[l] = diffusivity(w, q, Dw, Dg);
        S.low[l] = domain_chf(p, w, q) < (Real)0.1;
        return in_domain(w, q, p);
    };
    const int l = lab_at(t & 7, (t >> 3) & 7, t >> 6);
    const bool inside = put(l, base + t);
    if (t < 6 * 64) {
        // cell (a, e) of face f: 0 x-, 1 x+, 2 y-, 3 y+, 4 z-, 5 z+
        const int f = t >> 6, a = t & 7, e = (t >> 3) & 7, d = f >> 1;
        const int in = (f & 1) ? kBS : -1, from = (f & 1) ? 0 : kBS - 1;
        const int x = d == 0 ? in : a, y = d == 1 ? in : d == 0 ? a : e, z = d == 2 ? in : e;
        const int sx = d == 0 ? from : x, sy = d == 1 ? from : y, sz = d == 2 ? from : z;
        const int step = (f & 1) ? 1 : bpd - 1;
        const int nx = d == 0 ? (bx + step) % bpd : bx, ny = d == 1 ? (by + step) % bpd : by,
                  nz = d == 2 ? (bz + step) % bpd : bz;
        put(lab_at(x, y, z), (int64_t)(nx + bpd * (ny + bpd * nz)) * kBS3 + sx + kBS * (sy + kBS * sz));
    }
    __syncthreads();
    const int n[6] = {l - 1, l + 1, l - kLab, l + kLab, l - kLab * kLab, l + kLab * kLab};
    const Real phi = S.phi[l];
    Real dphidt = (Real)0.;
    if (inside) {
        Real H[6], phn[6];
        bool low[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            H[k] = face_harmonic(S.df[n[k]], S.df[l]);
            phn[k] = S.phi[n[k]];
            low[k] = S.low[n[k]];
        }
        dphidt = cell_rhs_flags<Real>(H[0], H[1], H[2], H[3], H[4], H[5], low, phn, phi, rho, ih2);
    }
    phi_out[base + t] = cell_update(phi, dphidt, dt);
}

template <typename Real>
int static_step(int bpd, const void *pw, const void *pg, const void *phi_in, void *phi_out, double Dw, double Dg,
                double rho, double dt, cudaStream_t s)
{
    const double h = (double)(Real)(1.0 / (8.0 * bpd));
    static_step_kernel<Real><<<bpd * bpd * bpd, kBS3, 0, s>>>(
        bpd, (const Real *)pw, (const Real *)pg, (const Real *)phi_in, (Real *)phi_out, (Real)Dw, (Real)Dg, (Real)rho,
        1. / (h * h), dt);
    return cudaGetLastError() == cudaSuccess ? GBFK_OK : GBFK_E_CUDA;
}

// Restores the caller's current device when the entry point returns.
struct DeviceGuard {
    int saved = -1;
    DeviceGuard() { if (cudaGetDevice(&saved) != cudaSuccess) saved = -1; }
    ~DeviceGuard() { if (saved >= 0) cudaSetDevice(saved); }
};

}  // namespace
}  // namespace gbfk

extern "C" int gbfk_rd_step_static(int precision, int bpd, const void *pw, const void *pg, const void *phi_in,
                                   void *phi_out, double Dw, double Dg, double rho, double dt, void *stream,
                                   int device)
{
    using namespace gbfk;
    if (precision != GBFK_F64 && precision != GBFK_F32) return GBFK_E_INVALID;
    if (bpd <= 0) return GBFK_E_INVALID;
    if ((long long)bpd * bpd * bpd > GBFK_STATIC_MAX_BLOCKS) return GBFK_E_TOO_LARGE;
    if (!pw || !pg || !phi_in || !phi_out) return GBFK_E_INVALID;
    // phi_out must not overlap phi_in anywhere: the step reads neighbours'
    // halos from phi_in while other CTAs write phi_out
    const uintptr_t bytes = (uintptr_t)bpd * bpd * bpd * 512 * (precision == GBFK_F64 ? 8 : 4);
    const uintptr_t in0 = (uintptr_t)phi_in, out0 = (uintptr_t)phi_out;
    if (in0 < out0 + bytes && out0 < in0 + bytes) return GBFK_E_INVALID;
    DeviceGuard guard;
    if (cudaSetDevice(device) != cudaSuccess) return GBFK_E_CUDA;
    // an error left pending by the caller's own earlier work is reported and
    // left in place, so that the launch checks below see only this call's
    if (cudaPeekAtLastError() != cudaSuccess) return GBFK_E_CUDA;
    cudaStream_t s = (cudaStream_t)stream;
    if (s) {
        // the stream must belong to `device`
        int sdev = -1;
        if (cudaStreamGetDevice(s, &sdev) != cudaSuccess || sdev != device) return GBFK_E_INVALID;
    }
    return precision == GBFK_F64 ? static_step<double>(bpd, pw, pg, phi_in, phi_out, Dw, Dg, rho, dt, s)
                                 : static_step<float>(bpd, pw, pg, phi_in, phi_out, Dw, Dg, rho, dt, s);
}
