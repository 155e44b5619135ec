// Device helpers of the kernels that keep blocks resident in shared memory:
// the forward runs (gbfk_resident.cu) and the adjoint runs
// (gbfk_resident_adjoint.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <type_traits>
#include <vector>

#include "gbfk_exact.cuh"
#include "gbfk_kernels.cuh"

namespace gbfk {
namespace {

constexpr unsigned long long kPollNs = 1000000000ull;  // a face not seen after 1 s is declared lost
constexpr unsigned kErrPoll = 1u | 512u;               // error word: a wait gave up, in a resident run

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// One thread's wait until `arrived` counts `target` arrivals (its own among
// them); false when that took longer than limit_ns.
__device__ __forceinline__ bool arrive_and_wait(unsigned *arrived, unsigned target, unsigned long long limit_ns)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
    unsigned long long since = 0;
    for (unsigned n = 0;; n++) {
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
        if (seen >= target) return true;
        if ((n & 1023u) == 1023u) {
            const unsigned long long now = now_ns();
            if (!since) since = now;
            else if (now - since > limit_ns) return false;
        }
    }
}

// ---- words of the exchange buffer -----------------------------------------
// N consecutive values in 16-, 8- or 4-byte accesses, each value one relaxed
// access of its own (no order among them is needed: each carries its phase)
template <int N>
__device__ __forceinline__ void ld_face(const float *p, float (&v)[N])
{
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3])
                         : "l"(p + i)
                         : "memory");
    } else
        asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p) : "memory");
}
template <int N>
__device__ __forceinline__ void ld_face(const double *p, double (&v)[N])
{
#pragma unroll
    for (int i = 0; i < N; i += 2)
        asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];"
                     : "=d"(v[i]), "=d"(v[i + 1])
                     : "l"(p + i)
                     : "memory");
}
template <int N>
__device__ __forceinline__ void st_face(float *p, const float (&v)[N])
{
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + i), "f"(v[i]), "f"(v[i + 1]),
                         "f"(v[i + 2]), "f"(v[i + 3])
                         : "memory");
    } else
        asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v[0]), "f"(v[1]) : "memory");
}
template <int N>
__device__ __forceinline__ void st_face(double *p, const double (&v)[N])
{
#pragma unroll
    for (int i = 0; i < N; i += 2)
        asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p + i), "d"(v[i]), "d"(v[i + 1]) : "memory");
}
__device__ __forceinline__ void st_face1(float *p, float v)
{
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_face1(double *p, double v)
{
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
// value with the sign bit set to the phase (m: the sign bit or 0), in one
// instruction the compiler does not see through: written with bit operators it
// becomes +-|v| in floating point, which drops the sign of a NaN
__device__ __forceinline__ unsigned with_phase_bits(unsigned v, unsigned m)
{
    unsigned r;
    asm("lop3.b32 %0, %1, 0x7fffffff, %2, 0xEA;" : "=r"(r) : "r"(v), "r"(m));  // (v & 0x7fffffff) | m
    return r;
}
__device__ __forceinline__ float with_phase(float v, unsigned m)
{
    return __uint_as_float(with_phase_bits(__float_as_uint(v), m));
}
__device__ __forceinline__ double with_phase(double v, unsigned m)
{
    return __hiloint2double((int)with_phase_bits((unsigned)__double2hiint(v), m), __double2loint(v));
}
// the sign bit differs from the phase: not there yet
__device__ __forceinline__ unsigned sign_xor(float v, unsigned m) { return __float_as_uint(v) ^ m; }
__device__ __forceinline__ unsigned sign_xor(double v, unsigned m) { return (unsigned)__double2hiint(v) ^ m; }
__device__ __forceinline__ float magnitude(float v) { return __uint_as_float(__float_as_uint(v) & 0x7fffffffu); }
__device__ __forceinline__ double magnitude(double v)
{
    return __hiloint2double(__double2hiint(v) & 0x7fffffff, __double2loint(v));
}

// The cells of a block are held by kT = 512 / kC threads, kC x-consecutive
// cells each.  Arrays in shared memory keep 16-byte vectors (or all kC cells,
// if they are fewer) as [vector][thread], so that a warp's access is one
// contiguous run of banks for every neighbour offset; rows of a face array
// count as threads too (kRows rows of 8).
template <typename Real, int kC, int kMaxV = 16 / (int)sizeof(Real)>
struct Tile {
    static constexpr int V = kMaxV < kC ? kMaxV : kC;
    // where cell x of a row lies in an array of kRows rows
    template <int kRows>
    static __device__ __forceinline__ int at(int row, int x)
    {
        const int t = row * (8 / kC) + x / kC, v = (x % kC) / V;
        return (v * (kRows * 8 / kC) + t) * V + x % V;
    }
    // the kC cells of "thread" t of such an array
    template <int kRows>
    static __device__ __forceinline__ void load(const Real *a, int t, Real (&d)[kC])
    {
#pragma unroll
        for (int v = 0; v < kC / V; v++) {
            const Real *p = a + (v * (kRows * 8 / kC) + t) * V;
            if constexpr (sizeof(Real) == 4 && V == 4) {
                const float4 q = *reinterpret_cast<const float4 *>(p);
                d[4 * v] = q.x; d[4 * v + 1] = q.y; d[4 * v + 2] = q.z; d[4 * v + 3] = q.w;
            } else if constexpr (sizeof(Real) == 4) {
                const float2 q = *reinterpret_cast<const float2 *>(p);
                d[2 * v] = q.x; d[2 * v + 1] = q.y;
            } else {
                const double2 q = *reinterpret_cast<const double2 *>(p);
                d[2 * v] = q.x; d[2 * v + 1] = q.y;
            }
        }
    }
    // pair v of thread t of an array with two-value vectors
    template <int kRows>
    static __device__ __forceinline__ int at2(int t, int v)
    {
        static_assert(V == 2, "pairs");
        return (v * (kRows * 8 / kC) + t) * 2;
    }
    template <int kRows>
    static __device__ __forceinline__ void load2(const Real *a, int t, int v, Real (&d)[2])
    {
        const Real *p = a + at2<kRows>(t, v);
        if constexpr (sizeof(Real) == 4) {
            const float2 q = *reinterpret_cast<const float2 *>(p);
            d[0] = q.x; d[1] = q.y;
        } else {
            const double2 q = *reinterpret_cast<const double2 *>(p);
            d[0] = q.x; d[1] = q.y;
        }
    }
    template <int kRows>
    static __device__ __forceinline__ void store(Real *a, int t, const Real (&d)[kC])
    {
#pragma unroll
        for (int v = 0; v < kC / V; v++) {
            Real *p = a + (v * (kRows * 8 / kC) + t) * V;
            if constexpr (sizeof(Real) == 4 && V == 4)
                *reinterpret_cast<float4 *>(p) = make_float4(d[4 * v], d[4 * v + 1], d[4 * v + 2], d[4 * v + 3]);
            else if constexpr (sizeof(Real) == 4)
                *reinterpret_cast<float2 *>(p) = make_float2(d[2 * v], d[2 * v + 1]);
            else
                *reinterpret_cast<double2 *>(p) = make_double2(d[2 * v], d[2 * v + 1]);
        }
    }
};
// kC consecutive cells of a block in global memory (16-byte aligned, or 8 for two floats)
template <typename Real, int kC>
__device__ __forceinline__ void ld_cells(const Real *p, Real (&d)[kC])
{
#pragma unroll
    for (int v = 0; v < kC / Tile<Real, kC>::V; v++) {
        constexpr int V = Tile<Real, kC>::V;
        if constexpr (sizeof(Real) == 4 && V == 4) {
            const float4 q = *reinterpret_cast<const float4 *>(p + 4 * v);
            d[4 * v] = q.x; d[4 * v + 1] = q.y; d[4 * v + 2] = q.z; d[4 * v + 3] = q.w;
        } else if constexpr (sizeof(Real) == 4) {
            const float2 q = *reinterpret_cast<const float2 *>(p + 2 * v);
            d[2 * v] = q.x; d[2 * v + 1] = q.y;
        } else {
            const double2 q = *reinterpret_cast<const double2 *>(p + 2 * v);
            d[2 * v] = q.x; d[2 * v + 1] = q.y;
        }
    }
}
template <typename Real, int kC>
__device__ __forceinline__ void st_cells(Real *p, const Real (&d)[kC])
{
    // consecutive vectors: a one-thread array
#pragma unroll
    for (int v = 0; v < kC / Tile<Real, kC>::V; v++) {
        constexpr int V = Tile<Real, kC>::V;
        if constexpr (sizeof(Real) == 4 && V == 4)
            *reinterpret_cast<float4 *>(p + 4 * v) = make_float4(d[4 * v], d[4 * v + 1], d[4 * v + 2], d[4 * v + 3]);
        else if constexpr (sizeof(Real) == 4)
            *reinterpret_cast<float2 *>(p + 2 * v) = make_float2(d[2 * v], d[2 * v + 1]);
        else
            *reinterpret_cast<double2 *>(p + 2 * v) = make_double2(d[2 * v], d[2 * v + 1]);
    }
}

// The state of a block with its face halos: rows y = -1 .. 8 of planes z = -1 ..
// 8, and the x faces apart.
constexpr int kRows = 100;
template <typename Real>
struct alignas(16) ResidentState {
    Real phi[kRows * 8];
    Real xh[2][64];          // [z][y]: the x- and x+ neighbours' cells
};
// What the cells of a warp need (two bits per warp of a block's threads):
//   kPlain    every cell and neighbour is kTissue: no no-flux doubling, every
//             cell is inside the domain;
//   kEdge     kEmpty cells or neighbours among them.  The coefficient of a
//             face that touches a kEmpty cell is 0, so its sign bit says so
//             (-0): a neighbour with phi < 0.1 across such a face doubles the
//             opposite coefficient (for a kEmpty cell itself, whose
//             coefficients are all 0, whatever is doubled stays 0, and its
//             formula leaves +0 where phi is +0 and the reaction where it is
//             not, so that its domain test needs no branch).  -0 for +0 in
//             the flux sums gives the same sums: (+0) + (-0) = +0 either way.
//             With a NaN among the neighbours that formula gives NaN where the
//             test keeps +0: the steps of a state with a NaN in it are not
//             these kernels' (see settle_kernel);
//   kGeneral  kOther cells or neighbours, or a coefficient that is negative
//             by itself: the tests as written, p_w and p_g from global memory;
//   kStill    kEmpty cells that hold +0, which stay so: nothing flows into a
//             kEmpty cell and +0 does not react. An eighth (128^3) to a
//             quarter (64^3) of the warps of a brain's heavy blocks.
constexpr unsigned kPlain = 0, kEdge = 1, kGeneral = 2, kStill = 3;

__device__ __forceinline__ float set_sign(float v, bool s) { return s ? __uint_as_float(__float_as_uint(v) | 0x80000000u) : v; }
__device__ __forceinline__ double set_sign(double v, bool s) { return s ? -v : v; }
__device__ __forceinline__ bool sign_of(float v) { return __float_as_int(v) < 0; }
__device__ __forceinline__ bool sign_of(double v) { return __double2hiint(v) < 0; }

// d = a * b and d += a for two values, each rounded to nearest by itself; one
// instruction for two floats.  The product is an FMA with -0 (which adds
// nothing, signs of zero included), and that -0 (neg0: both halves) comes
// from the host: the assembler contracts a packed multiply, or a packed FMA
// with a -0 it can see, with the packed add that follows.
__device__ __forceinline__ unsigned long long packed(const float (&v)[2])
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v[0]), "f"(v[1]));
    return r;
}
__device__ __forceinline__ void pair_mul(float (&d)[2], const float (&a)[2], const float (&b)[2],
                                         unsigned long long neg0)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(packed(a)), "l"(packed(b)), "l"(neg0));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d[0]), "=f"(d[1]) : "l"(r));
}
__device__ __forceinline__ void pair_add(float (&d)[2], const float (&a)[2])
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(packed(d)), "l"(packed(a)));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d[0]), "=f"(d[1]) : "l"(r));
}
__device__ __forceinline__ void pair_mul(double (&d)[2], const double (&a)[2], const double (&b)[2],
                                         unsigned long long)
{
    d[0] = rmul(a[0], b[0]);
    d[1] = rmul(a[1], b[1]);
}
__device__ __forceinline__ void pair_add(double (&d)[2], const double (&a)[2])
{
    d[0] = radd(d[0], a[0]);
    d[1] = radd(d[1], a[1]);
}
// clamp01 of a rounded result (its NaN is the canonical one): two instructions
__device__ __forceinline__ float clamp_state(float p)
{
    asm("max.NaN.f32 %0, %0, 0f00000000;" : "+f"(p));
    asm("min.NaN.f32 %0, %0, 0f3F800000;" : "+f"(p));
    return p;
}
__device__ __forceinline__ double clamp_state(double p) { return clamp01(p); }

// The pool blocks across the faces of block blk of the uniform periodic bpd^3 grid.
__device__ __forceinline__ int block_across(int bpd, int blk, int f)
{
    int q[3] = {blk % bpd, (blk / bpd) % bpd, blk / (bpd * bpd)};
    const int v = q[f >> 1] + ((f & 1) ? 1 : -1);
    q[f >> 1] = v < 0 ? bpd - 1 : v == bpd ? 0 : v;
    return q[0] + bpd * (q[1] + bpd * q[2]);
}

// What a thread needs to know of its place in a block, fixed for the run.
struct Place {
    int t;        // thread of the group
    int tp;       // its place in the padded state array
    int ty;       // its place in hy
    int xl, xr;   // element offsets in ResidentState of the cells before and after its own
    int he;       // element offset from hx of the last cell's right face
};
template <typename Real, int kC>
__device__ __forceinline__ Place place_of(int t)
{
    using TL = Tile<Real, kC, 2>;
    constexpr int R = 8 / kC;  // threads of a row
    const int x0 = (t % R) * kC, y = (t / R) & 7, z = t / (8 * R);
    const int row = z * 8 + y, prow = (z + 1) * 10 + y + 1;
    Place w;
    w.t = t;
    w.tp = prow * R + x0 / kC;
    w.ty = t + z * R;  // row z * 9 + y
    w.xl = x0 ? TL::template at<kRows>(prow, x0 - 1) : kRows * 8 + row;
    w.xr = x0 + kC < 8 ? TL::template at<kRows>(prow, x0 + kC) : kRows * 8 + 64 + row;
    w.he = x0 + kC < 8 ? Tile<Real, kC, 2>::template at<64>(row, x0 + kC) : kBS3 + row;
    return w;
}

// The no-flux tests of the pair of cells i, i + 1 of a thread of a clamped state
// (low[j][k]: neighbour k has chf < 0.1) and whether they are inside the
// domain (dom). kGeneral evaluates the tests as they are written, with p_w
// and p_g of the row and its neighbours from global memory; its loads do not
// wait for one another. (One load per cell that is kOther, each behind the
// test that finds it: 26 us per step for a 128^3 FP32 brain with a partial
// volume rim, of which 3 cells in 1000 are kOther.)
template <typename Real, int kC, unsigned kKind, typename Args, typename Block>
__device__ __forceinline__ void no_flux_tests(const Args &a, const Block &b, int t, int i, const Real (&ph)[2],
                                              const Real (&phn)[6][2], const Real (&df)[6][2], bool (&low)[2][6],
                                              bool (&dom)[2])
{
    const Real eps = (Real)0.1;
    if constexpr (kKind != kGeneral) {
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int k = 0; k < 6; k++) low[j][k] = kKind == kEdge && sign_of(df[k][j]) && phn[k][j] < eps;
    } else {
        constexpr int R = 8 / kC;
        const int x0 = (t % R) * kC, y = (t / R) & 7, z = t / (8 * R), row = z * 8 + y, c = t * kC + i;
        auto cell = [&](int f, int in) { return (int64_t)(f < 0 ? b.e >> 2 : b.at[f]) * kBS3 + in; };
        const int64_t at[6] = {i || x0 ? cell(-1, c - 1) : cell(0, row * 8 + 7),
                               i + 2 < kC || x0 + kC < 8 ? cell(-1, c + 2) : cell(1, row * 8),
                               y ? cell(-1, c - 8) : cell(2, c + 56),
                               y < 7 ? cell(-1, c + 8) : cell(3, c - 56),
                               z ? cell(-1, c - 64) : cell(4, c + 448),
                               z < 7 ? cell(-1, c + 64) : cell(5, c - 448)};
        Real w[6][2], g[6][2], ow[2], og[2];
        ld_cells(a.pw + cell(-1, c), ow);
        ld_cells(a.pg + cell(-1, c), og);
        w[0][0] = a.pw[at[0]];
        g[0][0] = a.pg[at[0]];
        w[1][1] = a.pw[at[1]];
        g[1][1] = a.pg[at[1]];
#pragma unroll
        for (int k = 2; k < 6; k++) {
            ld_cells(a.pw + at[k], w[k]);
            ld_cells(a.pg + at[k], g[k]);
        }
        w[0][1] = ow[0]; g[0][1] = og[0];
        w[1][0] = ow[1]; g[1][0] = og[1];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            dom[j] = in_domain(ow[j], og[j], ph[j]);
#pragma unroll
            for (int k = 0; k < 6; k++) low[j][k] = domain_chf(phn[k][j], w[k][j], g[k][j]) < eps;
        }
    }
}

// The coefficients of a block into shared memory (members hx, hx8, hy, hz of b,
// their signs set as kEdge says) and the kinds of its warps, by the block's
// kBS3 / kC threads together (sync: their barrier, taken once).  H, meta: the
// block's own.
template <typename Real, int kC, typename Block, typename Sync>
__device__ __forceinline__ void load_coefficients(Block &b, const Real *H, const unsigned short *meta, int t,
                                                  bool zero, Sync &&sync)
{
    using TL = Tile<Real, kC, 2>;
    constexpr int kT = kBS3 / kC;
    // face f along a direction touches a kEmpty cell: the cell after it is
    // kEmpty or has a kEmpty neighbour before it (the last face: the cell
    // before it, and its neighbour after it)
    auto touches = [&](int cell, int nb) { return (meta[cell] & 3u) == kEmpty || ((meta[cell] >> (2 + nb)) & 1u); };
    for (int q = t; q < 576; q += kT) {
        {
            const int f = q % 9, row = q / 9;
            const Real h = set_sign(H[q], f < 8 ? touches(row * 8 + f, 0) : touches(row * 8 + 7, 1));
            if (f < 8) b.hx[TL::template at<64>(row, f)] = h;
            else b.hx8[row] = h;
        }
        {
            const int x = q & 7, f = (q >> 3) % 9, zz = q / 72, row = q >> 3;
            b.hy[TL::template at<72>(row, x)] =
                set_sign(H[576 + q], f < 8 ? touches(zz * 64 + f * 8 + x, 2) : touches(zz * 64 + 56 + x, 3));
        }
        {
            const int x = q & 7, yy = (q >> 3) & 7, f = q >> 6, row = q >> 3;
            b.hz[TL::template at<72>(row, x)] =
                set_sign(H[1152 + q], f < 8 ? touches(f * 64 + yy * 8 + x, 4) : touches(448 + yy * 8 + x, 5));
        }
    }
    if (t == 0) b.kinds = 0;
    sync();
    unsigned kind = kPlain;
    bool still = zero;
    for (int i = 0; i < kC; i++) {
        const int cell = t * kC + i, x = cell & 7, row = cell >> 3, z = cell >> 6;
        const unsigned m = meta[cell];
        still = still && (m & 3u) == kEmpty;
        if ((m & 3u) == kOther || (m >> 8)) kind = kGeneral;
        else if (m != kMetaAllTissue && kind == kPlain) kind = kEdge;
        // a coefficient that is negative by itself (a negative tissue
        // fraction) has a sign that says nothing of kEmpty cells
        const Real d[6] = {b.hx[TL::template at<64>(row, x)], x < 7 ? b.hx[TL::template at<64>(row, x + 1)] : b.hx8[row],
                           b.hy[TL::template at<72>(row + z, x)], b.hy[TL::template at<72>(row + z + 1, x)],
                           b.hz[TL::template at<72>(row, x)], b.hz[TL::template at<72>(row + 8, x)]};
        for (int k = 0; k < 6; k++)
            if (sign_of(d[k]) != ((m & 3u) == kEmpty || ((m >> (2 + k)) & 1u))) kind = kGeneral;
    }
    const bool general = __any_sync(0xffffffffu, kind == kGeneral), edge = __any_sync(0xffffffffu, kind == kEdge);
    const bool all_still = __all_sync(0xffffffffu, still);
    if ((t & 31) == 0)
        atomicOr(&b.kinds, (all_still ? kStill : general ? kGeneral : edge ? kEdge : kPlain) << (2 * (t >> 5)));
}

// The kC cells p of a thread in block b (hx, hx8, hy, hz, e and at as
// in ResidentBlock) of a clamped state to out; xl, xr: the cells before and after
// them; rows(i, y0, y1, z0, z1): the neighbours of pair i; kKind: the cells of
// the thread's warp (kPlain, kEdge or kGeneral).
template <typename Real, int kC, unsigned kKind, typename Args, typename Block, typename Rows>
__device__ __forceinline__ void row_cells(const Args &a, double ih2, unsigned long long neg0, const Block &b,
                                          const Place &w, const Real (&p)[kC], Real xl, Real xr, Rows &&rows,
                                          Real (&out)[kC])
{
    using TL = Tile<Real, kC, 2>;
    constexpr int R = 8 / kC;  // threads of a row
    constexpr bool kLow = kKind != kPlain;
    // two cells at a time, so that the single-precision operations of the flux
    // sums can go in pairs (pair_add, pair_mul: each half rounded by itself),
    // and only one pair's coefficients are held at once
#pragma unroll
    for (int i = 0; i < kC; i += 2) {
        const Real ph[2] = {p[i], p[i + 1]};
        const Real xm[2] = {i ? p[i - 1] : xl, p[i]}, xp[2] = {p[i + 1], i + 2 < kC ? p[i + 2] : xr};
        Real d0[2], d1[2], d2[2], d3[2], d4[2], d5[2];
        TL::template load2<64>(b.hx, w.t, i / 2, d0);
        d1[0] = d0[1];
        d1[1] = i + 2 < kC ? b.hx[TL::template at2<64>(w.t, i / 2 + 1)] : b.hx[w.he];
        TL::template load2<72>(b.hy, w.ty, i / 2, d2);
        TL::template load2<72>(b.hy, w.ty + R, i / 2, d3);
        TL::template load2<72>(b.hz, w.t, i / 2, d4);
        TL::template load2<72>(b.hz, w.t + 8 * R, i / 2, d5);
        Real y0[2], y1[2], z0[2], z1[2];
        rows(i / 2, y0, y1, z0, z1);
        bool dom[2] = {true, true};
        if (kLow) {
            const Real phn[6][2] = {{xm[0], xm[1]}, {xp[0], xp[1]}, {y0[0], y0[1]},
                                    {y1[0], y1[1]}, {z0[0], z0[1]}, {z1[0], z1[1]}};
            const Real df[6][2] = {{d0[0], d0[1]}, {d1[0], d1[1]}, {d2[0], d2[1]},
                                   {d3[0], d3[1]}, {d4[0], d4[1]}, {d5[0], d5[1]}};
            bool lows[2][6];
            no_flux_tests<Real, kC, kKind>(a, b, w.t, i, ph, phn, df, lows, dom);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const bool (&low)[6] = lows[j];
                // _applyNoFluxBC: neighbour k below 0.1 doubles the opposite coefficient
                if (low[0]) d1[j] = rmul(d1[j], (Real)2.);
                if (low[1]) d0[j] = rmul(d0[j], (Real)2.);
                if (low[2]) d3[j] = rmul(d3[j], (Real)2.);
                if (low[3]) d2[j] = rmul(d2[j], (Real)2.);
                if (low[4]) d5[j] = rmul(d5[j], (Real)2.);
                if (low[5]) d4[j] = rmul(d4[j], (Real)2.);
            }
        }
        // cell_rhs: the same operations in the same order for both cells
        Real sin_[2] = {rmul(d0[0], xm[0]), rmul(d0[1], xm[1])}, u[2] = {rmul(d1[0], xp[0]), rmul(d1[1], xp[1])};
        pair_add(sin_, u);
        pair_mul(u, d2, y0, neg0);
        pair_add(sin_, u);
        pair_mul(u, d3, y1, neg0);
        pair_add(sin_, u);
        pair_mul(u, d4, z0, neg0);
        pair_add(sin_, u);
        pair_mul(u, d5, z1, neg0);
        pair_add(sin_, u);
        Real sdf[2] = {radd(d0[0], d1[0]), radd(d0[1], d1[1])};
        pair_add(sdf, d2);
        pair_add(sdf, d3);
        pair_add(sdf, d4);
        pair_add(sdf, d5);
        pair_mul(sdf, sdf, ph, neg0);
        const Real rr[2] = {a.rho, a.rho};
        Real rp[2];
        pair_mul(rp, rr, ph, neg0);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const double fluxIn = __dmul_rn(ih2, (double)sin_[j]);
            const double fluxOut = -__dmul_rn((double)sdf[j], ih2);
            const double phid = (double)ph[j];
            const double reaction = __dmul_rn((double)rp[j], __dadd_rn(1., -phid));
            const Real dphidt = to_real<Real>(__dadd_rn(__dadd_rn(fluxOut, fluxIn), reaction));
            const Real q = clamp_state(to_real<Real>(__dadd_rn(phid, __dmul_rn(a.dt, (double)dphidt))));
            out[i + j] = dom[j] ? q : ph[j];  // outside the domain a clamped value stays (dt is finite)
        }
        if (i + 2 < kC) asm volatile("" ::: "memory");
    }
}

constexpr int kMaxSmem = 227 * 1024;

// Raises a kernel's shared memory limit, once per device.
template <auto kernel>
cudaError_t raise_smem()
{
    static std::mutex mu;
    static std::vector<char> raised;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if ((int)raised.size() <= dev) raised.resize(dev + 1, 0);
    if (raised[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e == cudaSuccess) raised[dev] = 1;
    return e;
}
// A cooperative launch (CTAs wait for one another, so all must be resident).
template <auto kernel, typename... Args>
cudaError_t launch_coop(int ctas, int threads, size_t smem, cudaStream_t s, Args... args)
{
    if (smem > 48 * 1024) {
        const cudaError_t e = raise_smem<kernel>();
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) cudaGetLastError();  // reported here, not by the next launch's check
    return e;
}

}  // namespace
}  // namespace gbfk
