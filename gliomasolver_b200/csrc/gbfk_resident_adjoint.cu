// Runs of discrete adjoint steps with the blocks resident in shared memory
// (uniform grids whose heavy blocks fit).  The step is the one of
// adj_fused_kernel (gbfk_kernels.cu), with the same expressions in the same
// order: lambda_{k+1} of a cell from mu, the self term and the neighbours' mu of
// step k + 1 (phase A), then the forward step from phi_k, mu_k, the switch
// flags, the self term and the gradient terms of step k (phase B).
//
// One CTA per SM, launched cooperatively, as in gbfk_resident.cu: each heavy
// block belongs to one CTA for the run, and its mu, flags, self terms and face
// coefficients stay in shared memory.  phi_k and its halos come from the stored
// states (known before the launch, loaded one step ahead).  The faces of mu
// travel through L2 as 64-bit words that carry their own tag: mu has any sign,
// so a word is 32 bits of it and a step count, with one more bit that says
// whether the cell's coefficient across that face is doubled (FP64: two words).
// Two buffers are enough because of the group's barrier between the polls of a
// step and its stores (see gbfk_resident.cu).  Between launches mu, self terms
// and flags are kept in global memory, and each thread's compensated gradient
// sums too, so that the sums are the same bits however a sweep is cut into
// launches.
//
// What bounds it (128^3 FP32, 8 blocks per CTA, two rounds of four groups): 250
// warp instructions per 32 cells, 26 of them conversions between float and
// double, by 16 warps per SM that each wait on the dependent double-precision
// sums (45 % of the issue slots; 128 registers a thread allow no more warps).
// Measured on a B200: 8.2 us per adjoint step at 128^3 FP32 (14 with one launch
// per step), 4.7 at 64^3 FP64 (10); a 128^3 FP32 gradient of 1500 steps with 64
// checkpoints 34.6 -> 21.6 ms, with every state kept 29.4 -> 16.6, a 64^3 FP64
// one of 739 steps with 32 checkpoints 14.3 -> 6.7.
#include "gbfk_resident.cuh"

namespace gbfk {
namespace {

__device__ __forceinline__ void two_sum(double &s, double &c, double x)
{
    const double t = s + x;
    const double bp = t - s;
    c += (s - (t - bp)) + (x - bp);
    s = t;
}

// ---- words of the exchange buffer: (value bits, tag * 2 + doubled) ----------
// One 64-bit word for a float, two for a double, in 16-byte accesses where a
// thread has two words (each word by itself is complete: it carries its tag).
template <typename Real> struct Words { static constexpr int n = (int)sizeof(Real) / 4; };
__device__ __forceinline__ unsigned long long word_of(unsigned bits, unsigned tag)
{
    return (unsigned long long)tag << 32 | bits;
}
__device__ __forceinline__ void st_words(uint2 *p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words(const uint2 *p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_word(uint2 *p, float v, unsigned tag)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(word_of(__float_as_uint(v), tag)) : "memory");
}
__device__ __forceinline__ void st_word(uint2 *p, double v, unsigned tag)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    st_words(p, word_of((unsigned)b, tag), word_of((unsigned)(b >> 32), tag));
}
// two values with their own tags
__device__ __forceinline__ void st_word2(uint2 *p, const float *v, unsigned t0, unsigned t1)
{
    st_words(p, word_of(__float_as_uint(v[0]), t0), word_of(__float_as_uint(v[1]), t1));
}
__device__ __forceinline__ void st_word2(uint2 *p, const double *v, unsigned t0, unsigned t1)
{
    st_word(p, v[0], t0);
    st_word(p + 2, v[1], t1);
}
// two values, their tags, and the bits in which a tag differs from `tag` (shifted)
__device__ __forceinline__ unsigned ld_word2(const uint2 *p, float *v, unsigned *t, unsigned tag)
{
    unsigned long long a, b;
    ld_words(p, a, b);
    v[0] = __uint_as_float((unsigned)a);
    v[1] = __uint_as_float((unsigned)b);
    t[0] = (unsigned)(a >> 32);
    t[1] = (unsigned)(b >> 32);
    return (t[0] ^ tag) | (t[1] ^ tag);
}
__device__ __forceinline__ unsigned ld_word2(const uint2 *p, double *v, unsigned *t, unsigned tag)
{
    unsigned wrong = 0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        unsigned long long a, b;
        ld_words(p + 2 * i, a, b);
        v[i] = __longlong_as_double((long long)((a & 0xffffffffu) | b << 32));
        t[i] = (unsigned)(a >> 32);
        wrong |= (t[i] ^ tag) | ((unsigned)(b >> 32) ^ tag);
    }
    return wrong;
}

// Flags of a cell: bit 1 + k, its coefficient toward neighbour k is doubled
// (bit 0 as in adj_fused_kernel, unused here: a cell outside the domain has mu
// = 0).  [row][x] bytes with halos, then the x halos.
template <typename Real>
struct alignas(16) AdjBlock {
    ResidentState<Real> mu[2], phi[2];
    unsigned char fl[2][kRows * 8 + 128];
    double self[kBS3];
    Real hx[kBS3], hx8[64], hy[576], hz[576];
    int nbr[6], at[6];  // face neighbours: item (-1: an empty block), pool block
    int e;
    unsigned kinds;
};

// What the forward step from phi_k gives the adjoint step, for a thread's
// cells: the diffusive flux, the self term's factor, the switch flags, and
// whether the cell passes lambda on (0 < pre <= 1) and is inside the domain.
template <int kC>
struct AdjForward {
    double flux[kC], factor[kC];
    unsigned flags[kC];
    unsigned pass, dom;  // a bit per cell
};

// The two cells i, i + 1 of a thread, forward.
template <typename Real, int kC, unsigned kKind>
__device__ __forceinline__ void adj_forward(const AdjRunArgs<Real> &a, double ih2, unsigned long long neg0,
                                            const AdjBlock<Real> &b, const ResidentState<Real> &P, const Place &w, int i,
                                            AdjForward<kC> &out)
{
    using TL = Tile<Real, kC, 2>;
    constexpr int R = 8 / kC;
    Real d0[2], d1[2], d2[2], d3[2], d4[2], d5[2];
    TL::template load2<64>(b.hx, w.t, i / 2, d0);
    d1[0] = d0[1];
    d1[1] = i + 2 < kC ? b.hx[TL::template at2<64>(w.t, i / 2 + 1)] : b.hx[w.he];
    TL::template load2<72>(b.hy, w.ty, i / 2, d2);
    TL::template load2<72>(b.hy, w.ty + R, i / 2, d3);
    TL::template load2<72>(b.hz, w.t, i / 2, d4);
    TL::template load2<72>(b.hz, w.t + 8 * R, i / 2, d5);
    Real ph[2], y0[2], y1[2], z0[2], z1[2];
    TL::template load2<kRows>(P.phi, w.tp, i / 2, ph);
    TL::template load2<kRows>(P.phi, w.tp - R, i / 2, y0);
    TL::template load2<kRows>(P.phi, w.tp + R, i / 2, y1);
    TL::template load2<kRows>(P.phi, w.tp - 10 * R, i / 2, z0);
    TL::template load2<kRows>(P.phi, w.tp + 10 * R, i / 2, z1);
    const Real xm[2] = {P.phi[i == 0 ? w.xl : TL::template at2<kRows>(w.tp, i / 2 - 1) + 1], ph[0]},
               xp[2] = {ph[1], P.phi[i + 2 == kC ? w.xr : TL::template at2<kRows>(w.tp, i / 2 + 1)]};
    bool dom[2] = {true, true};
    unsigned fl[2] = {0, 0};
    if (kKind != kPlain) {
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
            if (low[0]) { d1[j] = rmul(d1[j], (Real)2.); fl[j] |= 4u; }
            if (low[1]) { d0[j] = rmul(d0[j], (Real)2.); fl[j] |= 2u; }
            if (low[2]) { d3[j] = rmul(d3[j], (Real)2.); fl[j] |= 16u; }
            if (low[3]) { d2[j] = rmul(d2[j], (Real)2.); fl[j] |= 8u; }
            if (low[4]) { d5[j] = rmul(d5[j], (Real)2.); fl[j] |= 64u; }
            if (low[5]) { d4[j] = rmul(d4[j], (Real)2.); fl[j] |= 32u; }
        }
    }
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
    Real sd[2] = {radd(d0[0], d1[0]), radd(d0[1], d1[1])};
    pair_add(sd, d2);
    pair_add(sd, d3);
    pair_add(sd, d4);
    pair_add(sd, d5);
    pair_mul(sd, sd, ph, neg0);
    const Real rr[2] = {a.rho, a.rho};
    Real rp[2];
    pair_mul(rp, rr, ph, neg0);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const double phd = (double)ph[j];
        const double fluxIn = __dmul_rn(ih2, (double)sin_[j]);
        const double fluxOut = -__dmul_rn((double)sd[j], ih2);
        const double reaction = __dmul_rn((double)rp[j], __dadd_rn(1., -phd));
        const Real dphidt = dom[j] ? to_real<Real>(__dadd_rn(__dadd_rn(fluxOut, fluxIn), reaction)) : (Real)0.;
        double sdf = 0;
        sdf += (double)d0[j];
        sdf += (double)d1[j];
        sdf += (double)d2[j];
        sdf += (double)d3[j];
        sdf += (double)d4[j];
        sdf += (double)d5[j];
        const Real pre = to_real<Real>(__dadd_rn(phd, __dmul_rn(a.dt, (double)dphidt)));
        out.flux[i + j] = fluxOut + fluxIn;
        out.factor[i + j] = -ih2 * sdf + (double)a.rho * (1. - 2. * phd);
        out.flags[i + j] = fl[j];
        if (pre > (Real)0 && pre <= (Real)1) out.pass |= 1u << (i + j);
        if (dom[j]) out.dom |= 1u << (i + j);
    }
}

// The flags of the neighbours of a thread's cells, a byte per cell, only the bit
// of the face between (see adj_lambda); any: one of them is set.
template <int kC>
struct AdjDoubling {
    unsigned dir[6];
    unsigned any;
};
template <int kC>
__device__ __forceinline__ AdjDoubling<kC> adj_doubling(const unsigned char *F, int row, int prow, int x0)
{
    const int f0 = prow * 8 + x0;
    auto cells = [&](int at) -> unsigned {
        if constexpr (kC == 4) return *reinterpret_cast<const unsigned *>(F + at);
        else return *reinterpret_cast<const unsigned short *>(F + at);
    };
    const unsigned own = cells(f0);
    const unsigned l = F[x0 == 0 ? kRows * 8 + row : f0 - 1], r = F[x0 + kC == 8 ? kRows * 8 + 64 + row : f0 + kC];
    AdjDoubling<kC> d;
    // neighbour k doubles its coefficient k ^ 1 toward the cell: bit 1 + (k ^ 1)
    d.dir[0] = (own << 8 | l) & 0x04040404u;
    d.dir[1] = (own >> 8 | r << (8 * (kC - 1))) & 0x02020202u;
    d.dir[2] = cells(f0 - 8) & 0x10101010u;
    d.dir[3] = cells(f0 + 8) & 0x08080808u;
    d.dir[4] = cells(f0 - 80) & 0x40404040u;
    d.dir[5] = cells(f0 + 80) & 0x20202020u;
    d.any = d.dir[0] | d.dir[1] | d.dir[2] | d.dir[3] | d.dir[4] | d.dir[5];
    return d;
}

// The two cells i, i + 1 of a thread: lambda of step k + 1 from mu, flags and
// self terms of that step.
template <typename Real, int kC>
__device__ __forceinline__ void adj_lambda(const AdjRunArgs<Real> &a, double ih2, const AdjBlock<Real> &b, int cur,
                                           const Place &w, const AdjDoubling<kC> &dbl, int i, Real (&lam)[2])
{
    using TL = Tile<Real, kC, 2>;
    constexpr int R = 8 / kC;
    Real d0[2], d1[2], d2[2], d3[2], d4[2], d5[2];
    TL::template load2<64>(b.hx, w.t, i / 2, d0);
    d1[0] = d0[1];
    d1[1] = i + 2 < kC ? b.hx[TL::template at2<64>(w.t, i / 2 + 1)] : b.hx[w.he];
    TL::template load2<72>(b.hy, w.ty, i / 2, d2);
    TL::template load2<72>(b.hy, w.ty + R, i / 2, d3);
    TL::template load2<72>(b.hz, w.t, i / 2, d4);
    TL::template load2<72>(b.hz, w.t + 8 * R, i / 2, d5);
    const ResidentState<Real> &M = b.mu[cur];
    Real m[2], y0[2], y1[2], z0[2], z1[2];
    TL::template load2<kRows>(M.phi, w.tp, i / 2, m);
    TL::template load2<kRows>(M.phi, w.tp - R, i / 2, y0);
    TL::template load2<kRows>(M.phi, w.tp + R, i / 2, y1);
    TL::template load2<kRows>(M.phi, w.tp - 10 * R, i / 2, z0);
    TL::template load2<kRows>(M.phi, w.tp + 10 * R, i / 2, z1);
    const Real xl = M.phi[i == 0 ? w.xl : TL::template at2<kRows>(w.tp, i / 2 - 1) + 1],
               xr = M.phi[i + 2 == kC ? w.xr : TL::template at2<kRows>(w.tp, i / 2 + 1)];
    double g[6][2] = {{(double)d0[0], (double)d0[1]}, {(double)d1[0], (double)d1[1]}, {(double)d2[0], (double)d2[1]},
                      {(double)d3[0], (double)d3[1]}, {(double)d4[0], (double)d4[1]}, {(double)d5[0], (double)d5[1]}};
    if (dbl.any) {
#pragma unroll
        for (int k = 0; k < 6; k++)
#pragma unroll
            for (int j = 0; j < 2; j++)
                if (dbl.dir[k] >> (8 * (i + j)) & 0xffu) g[k][j] *= 2.;
    }
    const Real xm[2] = {xl, m[0]}, xp[2] = {m[1], xr};
    const double2 sf = *reinterpret_cast<const double2 *>(b.self + (i / 2 * (kBS3 / kC) + w.t) * 2);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        double s = 0;
        s += j ? sf.y : sf.x;
        s += ih2 * g[0][j] * (double)xm[j];
        s += ih2 * g[1][j] * (double)xp[j];
        s += ih2 * g[2][j] * (double)y0[j];
        s += ih2 * g[3][j] * (double)y1[j];
        s += ih2 * g[4][j] * (double)z0[j];
        s += ih2 * g[5][j] * (double)z1[j];
        lam[j] = (Real)((double)m[j] + a.dt * s);
    }
}

// mu, the self term and the gradient terms of cell i of a thread.
template <typename Real, int kC, bool kAbs>
__device__ __forceinline__ Real adj_mu(const AdjRunArgs<Real> &a, const AdjForward<kC> &fw, int i, Real lam, Real ph,
                                       double &self, double (&acc)[6])
{
    const bool pass = fw.pass >> i & 1u, dom = fw.dom >> i & 1u;
    const Real mv = pass ? lam : (Real)0;
    const double mvd = (double)mv, phd = (double)ph;
    self = dom ? mvd * fw.factor[i] : 0.;
    if (dom && pass) {
        // dt and 1 / Dw are the caller's factors of the sums
        const double tr = mvd * (phd * (1. - phd));
        const double td = mvd * fw.flux[i];
        two_sum(acc[0], acc[1], tr);
        two_sum(acc[2], acc[3], td);
        if (kAbs) {
            acc[4] += fabs(tr);
            acc[5] += fabs(td);
        }
    }
    return mv;
}

constexpr int kHead = 768;  // bytes of shared memory before the blocks

template <typename Real, int kC, int kGroups, bool kAbs>
__global__ void __launch_bounds__(kGroups * (kBS3 / kC), 1)
adj_run_kernel(const __grid_constant__ AdjRunArgs<Real> a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AdjBlock<Real> *blocks = reinterpret_cast<AdjBlock<Real> *>(smem_raw + kHead);
    using TL = Tile<Real, kC, 2>;
    constexpr int kT = kBS3 / kC, R = 8 / kC, W = Words<Real>::n;
    const int t = threadIdx.x % kT, group = threadIdx.x / kT;
    const int c = blockIdx.x, G = gridDim.x;
    const int nlocal = a.n > c ? (a.n - 1 - c) / G + 1 : 0;
    const Place w = place_of<Real, kC>(t);
    const int x0 = (t % R) * kC, y = (t / R) & 7, z = t / (8 * R), row = z * 8 + y, prow = (z + 1) * 10 + y + 1;
    // the halo vector this thread fetches: kC cells of face pf from pw on
    constexpr bool kAll = kT * kC <= 384;
    const int pf = t * kC / 64, pw = (t * kC) % 64;
    const bool fetches = kAll || pf < 6;
    const int pstep = pf < 2 ? TL::V : kRows * 8 / kC * TL::V;
    const int prow_h = pf < 4 ? (pw / 8 + 1) * 10 + (pf == 2 ? 0 : 9) : (pf == 4 ? 0 : 90) + pw / 8 + 1;
    const int pd = pf < 2 ? kRows * 8 + pf * 64 + pw : TL::template at<kRows>(prow_h, pw % 8);
    const int pfl = pf < 2 ? kRows * 8 + pf * 64 + pw : prow_h * 8 + pw % 8;  // its flag bytes
    // where the halo vector starts in the neighbour block's 512 cells, and the
    // distance of its cells (face pf of this block is its face pf ^ 1)
    const int pc = pf == 0   ? pw * 8 + 7
                   : pf == 1 ? pw * 8
                   : pf < 4  ? (pw / 8) * 64 + (pf == 2 ? 56 : 0) + pw % 8
                             : (pf == 4 ? 448 : 0) + pw;
    const int pcs = pf < 2 ? 8 : 1;
    const unsigned tag0 = *a.index;  // faces stored by earlier launches
    auto buf = [&](unsigned tag) { return a.ex + (int64_t)((tag & 1u) ? a.n : 0) * 384 * W; };
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kT) : "memory"); };
    auto publish = [&](int item, const Real (&v)[kC], const unsigned (&f)[kC], unsigned tag) {
        uint2 *ex = buf(tag) + (int64_t)item * 384 * W;
        const unsigned t2 = tag << 1;
        if (x0 == 0) st_word(ex + row * W, v[0], t2 | (f[0] >> 1 & 1u));
        if (x0 + kC == 8) st_word(ex + (64 + row) * W, v[kC - 1], t2 | (f[kC - 1] >> 2 & 1u));
#pragma unroll
        for (int i = 0; i < kC; i += 2) {
            if (y == 0) st_word2(ex + (128 + z * 8 + x0 + i) * W, v + i, t2 | (f[i] >> 3 & 1u), t2 | (f[i + 1] >> 3 & 1u));
            if (y == 7) st_word2(ex + (192 + z * 8 + x0 + i) * W, v + i, t2 | (f[i] >> 4 & 1u), t2 | (f[i + 1] >> 4 & 1u));
            if (z == 0) st_word2(ex + (256 + y * 8 + x0 + i) * W, v + i, t2 | (f[i] >> 5 & 1u), t2 | (f[i + 1] >> 5 & 1u));
            if (z == 7) st_word2(ex + (320 + y * 8 + x0 + i) * W, v + i, t2 | (f[i] >> 6 & 1u), t2 | (f[i + 1] >> 6 & 1u));
        }
    };
    auto store_flags = [&](unsigned char *F, const unsigned (&f)[kC]) {
#pragma unroll
        for (int i = 0; i < kC; i += 2)
            *reinterpret_cast<unsigned short *>(F + prow * 8 + x0 + i) = (unsigned short)(f[i] | f[i + 1] << 8);
    };

    double acc[6] = {};
    double *my_acc = a.acc + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 6;
    if (!a.first)
#pragma unroll
        for (int i = 0; i < (kAbs ? 6 : 4); i++) acc[i] = my_acc[i];

    // the group's blocks into shared memory
    for (int j = group; j < nlocal; j += kGroups) {
        AdjBlock<Real> &b = blocks[j];
        const int item = c + j * G, e = a.items[item];
        const int64_t blk = e >> 2;
        if (t == 0) b.e = e;
        if (t < 6) {
            const int nb = a.nbr[item * 6 + t];
            b.nbr[t] = nb;
            b.at[t] = block_across(a.bpd, e >> 2, t);
        }
        if (fetches && a.nbr[item * 6 + pf] < 0)  // an empty neighbour: phi = mu = 0
            for (int s = 0; s < 2; s++)
                for (int v = 0; v < kC / TL::V; v++)
                    for (int i = 0; i < TL::V; i++) {
                        b.phi[s].phi[pd + v * pstep + i] = b.mu[s].phi[pd + v * pstep + i] = (Real)0;
                        b.fl[s][pfl + v * TL::V + i] = 0;
                    }
        if (!a.first) {
            Real v[kC];
            unsigned f[kC];
            ld_cells((const Real *)a.mu + (int64_t)item * kBS3 + t * kC, v);
            TL::template store<kRows>(b.mu[0].phi, w.tp, v);
#pragma unroll
            for (int i = 0; i < kC; i++) {
                f[i] = a.flags[(int64_t)item * kBS3 + t * kC + i];
                b.self[(i / 2 * kT + t) * 2 + (i & 1)] = a.self[(int64_t)item * kBS3 + t * kC + i];
            }
            store_flags(b.fl[0], f);
            publish(item, v, f, tag0 + 1);
        }
        load_coefficients<Real, kC>(b, a.H + blk * kFacesPerBlock, a.meta + blk * kBS3, t, false, group_sync);
    }
    group_sync();

    // phi of the next (step, block) of this group: its own cells and the halo
    // vector it fetches
    Real pn[kC], hn[kC];
    auto fetch_phi = [&](int s, int j) {
        if (s >= a.nsteps || j >= nlocal) return;
        const AdjBlock<Real> &b = blocks[j];
        const Real *phi = a.states[s];
        ld_cells(phi + (int64_t)(b.e >> 2) * kBS3 + t * kC, pn);
        if (fetches) {
            if (b.nbr[pf] >= 0) {
                const Real *q = phi + (int64_t)b.at[pf] * kBS3 + pc;
#pragma unroll
                for (int i = 0; i < kC; i++) hn[i] = q[i * pcs];
            }
        }
    };
    fetch_phi(0, group);
    const int passes = a.nsteps + (a.final ? 1 : 0);
    unsigned tag = tag0 + (a.first ? 0 : 1);  // the tag of the faces this pass reads (none in a first pass)
    bool failed = false;
    for (int s = 0; s < passes; s++) {
        const int cur = s & 1;
        const bool given = a.first && s == 0, last = s == a.nsteps;
        for (int j = group; j < nlocal; j += kGroups) {
            AdjBlock<Real> &b = blocks[j];
            const int item = c + j * G;
            if (!last) {
                TL::template store<kRows>(b.phi[cur].phi, w.tp, pn);
                if (fetches && b.nbr[pf] >= 0) {
#pragma unroll
                    for (int v = 0; v < kC / TL::V; v++) {
                        Real q[TL::V];
#pragma unroll
                        for (int i = 0; i < TL::V; i++) q[i] = hn[v * TL::V + i];
                        st_cells(b.phi[cur].phi + pd + v * pstep, q);
                    }
                }
            }
            const int64_t cell = (int64_t)(b.e >> 2) * kBS3 + t * kC;
            // the forward step, while the neighbours' faces are on their way
            AdjForward<kC> fw;
            fw.pass = fw.dom = 0;
            if (!last) {
                group_sync();
                if (j + kGroups < nlocal) fetch_phi(s, j + kGroups);
                else fetch_phi(s + 1, group);
                const unsigned kind = (b.kinds >> (2 * (t >> 5))) & 3u;
#pragma unroll
                for (int i = 0; i < kC; i += 2) {
                    if (kind == kPlain) adj_forward<Real, kC, kPlain>(a, a.ih2, a.neg0, b, b.phi[cur], w, i, fw);
                    else if (kind == kEdge) adj_forward<Real, kC, kEdge>(a, a.ih2, a.neg0, b, b.phi[cur], w, i, fw);
                    else adj_forward<Real, kC, kGeneral>(a, a.ih2, a.neg0, b, b.phi[cur], w, i, fw);
                }
            }
            if (!given && fetches && b.nbr[pf] >= 0) {
                const uint2 *src = buf(tag) + ((int64_t)b.nbr[pf] * 384 + (pf ^ 1) * 64 + pw) * W;
                Real h[kC];
                unsigned f[kC];
                unsigned long long t0 = 0;
                for (int it = 0;; it++) {
                    unsigned wrong = 0;
#pragma unroll
                    for (int i = 0; i < kC; i += 2) wrong |= ld_word2(src + i * W, h + i, f + i, tag << 1);
                    if (!(wrong & ~1u)) break;
                    if ((it & 63) == 63) {
                        if (t0 == 0) t0 = now_ns();
                        else if (now_ns() - t0 > kPollNs || it > (1 << 24)) {
                            failed = true;
                            break;
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < kC / TL::V; v++) {
                    Real q[TL::V];
#pragma unroll
                    for (int i = 0; i < TL::V; i++) {
                        q[i] = h[v * TL::V + i];
                        b.fl[cur][pfl + v * TL::V + i] = (unsigned char)((f[v * TL::V + i] & 1u) << (1 + (pf ^ 1)));
                    }
                    st_cells(b.mu[cur].phi + pd + v * pstep, q);
                }
            }
            unsigned any;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t"
                "setp.ne.u32 p, %1, 0;\n\t"
                "barrier.cta.red.or.pred q, %2, %3, p;\n\t"
                "selp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(any)
                : "r"((unsigned)failed), "r"(group + 1), "n"(kT)
                : "memory");
            if (any) {
                if (t == 0) atomicOr(a.err_flag, kErrPoll);
                goto out;
            }
            Real o[kC];
            AdjDoubling<kC> dbl = {};
            if (given) ld_cells(a.lam + cell, o);
            else dbl = adj_doubling<kC>(b.fl[cur], row, prow, x0);
#pragma unroll
            for (int i = 0; i < kC; i += 2) {
                Real l2[2] = {o[i], o[i + 1]};
                if (!given) adj_lambda<Real, kC>(a, a.ih2, b, cur, w, dbl, i, l2);
                if (!last) {
                    Real ph[2];
                    TL::template load2<kRows>(b.phi[cur].phi, w.tp, i / 2, ph);
                    double2 sf;
                    l2[0] = adj_mu<Real, kC, kAbs>(a, fw, i, l2[0], ph[0], sf.x, acc);
                    l2[1] = adj_mu<Real, kC, kAbs>(a, fw, i + 1, l2[1], ph[1], sf.y, acc);
                    *reinterpret_cast<double2 *>(b.self + (i / 2 * kT + t) * 2) = sf;
                }
                o[i] = l2[0];
                o[i + 1] = l2[1];
            }
            const unsigned(&f)[kC] = fw.flags;
            if (last) {
                st_cells(a.lam_out + cell, o);
                continue;
            }
            if (s + 1 < passes) {
                publish(item, o, f, tag + 1);
                TL::template store<kRows>(b.mu[cur ^ 1].phi, w.tp, o);
                store_flags(b.fl[cur ^ 1], f);
            } else {  // for the next launch
                st_cells((Real *)a.mu + (int64_t)item * kBS3 + t * kC, o);
#pragma unroll
                for (int i = 0; i < kC; i++) {
                    a.flags[(int64_t)item * kBS3 + t * kC + i] = (unsigned char)f[i];
                    a.self[(int64_t)item * kBS3 + t * kC + i] = b.self[(i / 2 * kT + t) * 2 + (i & 1)];
                }
            }
        }
        tag++;
    }
out:
    if (!a.final) {
#pragma unroll
        for (int i = 0; i < (kAbs ? 6 : 4); i++) my_acc[i] = acc[i];
    }
    // faces stored: one per pass but the last one, and the initial one
    static_assert(kGroups * kT / 32 * 6 * sizeof(double) <= kHead, "one row per warp");
    double(*red)[6] = reinterpret_cast<double(*)[6]>(smem_raw);
    if (a.final) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                const double s2 = __shfl_down_sync(0xffffffffu, acc[q], off), c2 = __shfl_down_sync(0xffffffffu, acc[q + 1], off);
                two_sum(acc[q], acc[q + 1], s2);
                acc[q + 1] += c2;
            }
            acc[4] += __shfl_down_sync(0xffffffffu, acc[4], off);
            acc[5] += __shfl_down_sync(0xffffffffu, acc[5], off);
        }
        if ((threadIdx.x & 31) == 0)
            for (int q = 0; q < 6; q++) red[threadIdx.x >> 5][q] = acc[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (a.final) {
            for (int v = 1; v < kGroups * kT / 32; v++) {
                for (int q = 0; q < 4; q += 2) {
                    two_sum(red[0][q], red[0][q + 1], red[v][q]);
                    red[0][q + 1] += red[v][q + 1];
                }
                red[0][4] += red[v][4];
                red[0][5] += red[v][5];
            }
            for (int q = 0; q < 6; q++) a.sums[blockIdx.x * 6 + q] = red[0][q];
        }
        if (atomicAdd(a.index + 1, 1u) == (unsigned)G - 1) {
            a.index[1] = 0;
            a.index[0] = (tag0 + (unsigned)passes) & 0x7fffffffu;
        }
    }
}

// Cells per thread and groups per CTA by the blocks of a CTA: 512 threads of up
// to 128 registers either way, two cells each while a block per group is all
// there is to do.  More groups spill (128^3 FP32, 8 blocks per CTA, 1500 steps
// with their forward steps on a B200: 16.6 ms with four groups of four cells,
// 20.0 with five, 23.3 with six, 18.8 with three groups of two cells).
template <typename Real, typename F>
cudaError_t adj_shape(int per, F &&f)
{
    using std::integral_constant;
    if (per <= 2) return f(integral_constant<int, 2>(), integral_constant<int, 2>());
    return f(integral_constant<int, 4>(), integral_constant<int, 4>());
}

}  // namespace

template <typename Real>
int adjoint_run_capacity(int sms)
{
    return sms * ((kMaxSmem - kHead) / (int)sizeof(AdjBlock<Real>));
}

int adjoint_run_threads(int n, int sms)
{
    const int ctas = n < sms ? n : sms;
    return ctas * 512;  // of either shape
}

template <typename Real>
cudaError_t launch_adjoint_run(const AdjRunArgs<Real> &a, bool abs_terms, int sms, cudaStream_t s)
{
    if (a.n <= 0 || a.nsteps < 0 || a.n > adjoint_run_capacity<Real>(sms)) return cudaErrorInvalidValue;
    const int ctas = a.n < sms ? a.n : sms, per = (a.n + ctas - 1) / ctas;
    const size_t smem = kHead + (size_t)per * sizeof(AdjBlock<Real>);
    return adj_shape<Real>(per, [&](auto c, auto g) {
        constexpr int kC = decltype(c)::value, kGroups = decltype(g)::value;
        constexpr int threads = kGroups * (kBS3 / kC);
        return abs_terms ? launch_coop<adj_run_kernel<Real, kC, kGroups, true>>(ctas, threads, smem, s, a)
                         : launch_coop<adj_run_kernel<Real, kC, kGroups, false>>(ctas, threads, smem, s, a);
    });
}

template int adjoint_run_capacity<float>(int);
template int adjoint_run_capacity<double>(int);
template cudaError_t launch_adjoint_run<float>(const AdjRunArgs<float> &, bool, int, cudaStream_t);
template cudaError_t launch_adjoint_run<double>(const AdjRunArgs<double> &, bool, int, cudaStream_t);

}  // namespace gbfk
