// The UQ end of the path: the finest-uniform dump of phi
// (Glioma_ReactionDiffusion::_dumpUQoutput, Glioma/Glioma_ReactionDiffusion.cpp:
// 208-262) and the log-likelihood of the observations
// (HGG_Likelihood.cpp:40-156 in tools/pi4u_lite/Inference/Likelihood/source),
// both on the device so that a TMCMC sample never leaves HBM.
#include "gbfk_exact.cuh"
#include "gbfk_kernels.cuh"

#include <algorithm>
#include <type_traits>

namespace gbfk {

// One thread per pool cell.  x = origin + h*i in Real (BlockInfo::pos,
// MRAG/MRAGcore/MRAGCommon.h:199), voxel m = floor(x / hf).  Blocks at least as
// fine as the dump grid write their voxel from the last cell that maps to it in
// the reference's z, y, x loop order; coarser blocks write c^3 copies with
// c = 2, 3 or 4 chosen by h exactly as the reference does.
template <typename Real>
__global__ void uq_dump_kernel(const int *__restrict__ slot, const Real *__restrict__ origin,
                               const Real *__restrict__ hblk, int nblocks, const Real *__restrict__ phi, int gpd,
                               double *__restrict__ out)
{
    const int64_t n = (int64_t)nblocks * kBS3;
    const double hf = 1. / gpd;
    const double eps = hf * 0.5;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(i >> 9), c = (int)(i & 511);
        const int ix = c & 7, iy = (c >> 3) & 7, iz = c >> 6;
        const Real hb = hblk[b];
        const Real o0 = origin[3 * b], o1 = origin[3 * b + 1], o2 = origin[3 * b + 2];
        const double x0 = radd(o0, rmul(hb, (Real)ix)), x1 = radd(o1, rmul(hb, (Real)iy)),
                     x2 = radd(o2, rmul(hb, (Real)iz));
        const int mx = (int)floor(__ddiv_rn(x0, hf)), my = (int)floor(__ddiv_rn(x1, hf)),
                  mz = (int)floor(__ddiv_rn(x2, hf));
        const double hd = hb;
        const double v = (double)phi[(int64_t)slot[b] * kBS3 + c];
        int cc;
        if (hd < hf + eps) {
            // last writer of the voxel in loop order: the next cell along each
            // direction maps to another voxel or lies outside the block
            const bool lx = ix == 7 || (int)floor(__ddiv_rn((double)radd(o0, rmul(hb, (Real)(ix + 1))), hf)) != mx;
            const bool ly = iy == 7 || (int)floor(__ddiv_rn((double)radd(o1, rmul(hb, (Real)(iy + 1))), hf)) != my;
            const bool lz = iz == 7 || (int)floor(__ddiv_rn((double)radd(o2, rmul(hb, (Real)(iz + 1))), hf)) != mz;
            if (!(lx && ly && lz)) continue;
            cc = 1;
        } else if (hd < 2. * hf + eps) cc = 2;
        else if (hd < 3. * hf + eps) cc = 3;
        else cc = 4;
        for (int cz = 0; cz < cc; cz++)
            for (int cy = 0; cy < cc; cy++)
                for (int cx = 0; cx < cc; cx++)
                    out[(mx + cx) + (int64_t)gpd * ((my + cy) + (int64_t)gpd * (mz + cz))] = v;
    }
}

template <typename Real>
cudaError_t launch_uq_dump(const int *slot, const Real *origin, const Real *hblk, int nblocks, const Real *phi,
                           int gpd, double *out, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double) * (size_t)gpd * gpd * gpd, s);
    if (e != cudaSuccess || nblocks <= 0) return e;
    int64_t nb = ((int64_t)nblocks * kBS3 + 255) / 256;
    if (nb > 148 * 32) nb = 148 * 32;
    uq_dump_kernel<Real><<<(int)nb, 256, 0, s>>>(slot, origin, hblk, nblocks, phi, gpd, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Log-likelihood terms with compensated (Neumaier) double sums.  The
// reference sums in long double; with compensation the device sums carry
// about 106 bits, and each term is the exact value of the reference's
// expression computed without cancellation:
//   alpha = 0.5 + 0.5*sgn(d)*(1 - exp(-t)),  t = omega2/slope,
//   omega2 = 1 if d > 0 else d^2,  d = u - uc       (HGG_Likelihood.cpp:149-155)
// so for d > 0: log(alpha) = log1p(-e/2), log(1-alpha) = log(1/2) - t,
//    for d < 0: log(alpha) = log(1/2) - t, log(1-alpha) = log1p(-e/2), e = exp(-t).
struct Neumaier {
    double s, c;
    __device__ void add(double x)
    {
        const double t = s + x;
        if (fabs(s) >= fabs(x)) c += (s - t) + x;
        else c += (x - t) + s;
        s = t;
    }
    __device__ void merge(const Neumaier &o)
    {
        add(o.s);
        add(o.c);
    }
};

// Sums of a CTA's threads, the same bits in every run: pairs (sum,
// compensation) and whole numbers, by warp shuffles, then warp by warp through
// shared memory; the result is thread 0's, the whole numbers in `total` (a warp's
// below 2^32).
template <int kPairs, int kCounts, int kWarps, typename Total>
__device__ __forceinline__ void cta_sums(Neumaier (&v)[kPairs], unsigned (&k)[kCounts],
                                         double (&red)[kWarps][2 * kPairs], unsigned (&cnt)[kWarps][kCounts],
                                         Total (&total)[kCounts])
{
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int i = 0; i < kPairs; i++) {
            Neumaier o;
            o.s = __shfl_down_sync(0xffffffffu, v[i].s, off);
            o.c = __shfl_down_sync(0xffffffffu, v[i].c, off);
            v[i].merge(o);
        }
#pragma unroll
    for (int i = 0; i < kCounts; i++) k[i] = __reduce_add_sync(0xffffffffu, k[i]);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < kPairs; i++) {
            red[w][2 * i] = v[i].s;
            red[w][2 * i + 1] = v[i].c;
        }
#pragma unroll
        for (int i = 0; i < kCounts; i++) cnt[w][i] = k[i];
    }
    __syncthreads();
    if (t != 0) return;
#pragma unroll
    for (int i = 0; i < kCounts; i++) total[i] = k[i];
    for (int j = 1; j < kWarps; j++) {
#pragma unroll
        for (int i = 0; i < kPairs; i++) v[i].merge(Neumaier{red[j][2 * i], red[j][2 * i + 1]});
#pragma unroll
        for (int i = 0; i < kCounts; i++) total[i] += cnt[j][i];
    }
}

__device__ __forceinline__ void bernoulli_terms(double u, double uc, double is2, double &log_a, double &log_1a)
{
    const double d = u - uc;
    const int sg = (d < -0.0) ? -1 : (d > 0.0 ? 1 : 0);
    const double t = (d > 0.) ? is2 : d * d * is2;
    const double lhalf = -0.69314718055994530942;  // log(1/2)
    if (sg == 0) {
        log_a = log_1a = lhalf;
    } else {
        const double e = exp(-t);
        const double a = log1p(-0.5 * e), b = lhalf - t;
        log_a = sg > 0 ? a : b;
        log_1a = sg > 0 ? b : a;
    }
}

// Where a state's values lie: the n^3 dump grid (doubles, x fastest), or the
// block pool of a uniform grid, whose dump is its own cells.  A thread reads
// kRow x-consecutive values at a time.
struct DenseState {
    static constexpr int kRow = 1;
    const double *u;
    __device__ double at(int n, int x, int y, int z) const { return u[x + (int64_t)n * (y + (int64_t)n * z)]; }
    __device__ void row(int64_t r, int, double (&v)[1]) const { v[0] = u[r]; }
    __device__ int offset_of_row(int64_t, int) const { return 0; }
};
template <typename Real>
struct PoolState {
    static constexpr int kRow = 8;
    const Real *u;
    __device__ double at(int n, int x, int y, int z) const
    {
        const int bpd = n >> 3;
        return (double)u[((x >> 3) + (int64_t)bpd * ((y >> 3) + (int64_t)bpd * (z >> 3))) * kBS3 + (x & 7) +
                         kBS * ((y & 7) + kBS * (z & 7))];
    }
    // row r of the dense grid: block column r % bpd of line (y, z)
    // (a pool has at most 2^31 cells)
    __device__ int offset_of_row(int64_t r, int n) const
    {
        const int bpd = n >> 3, line = (int)(r / bpd), bx = (int)(r - (int64_t)line * bpd), z = line / n, y = line - z * n;
        return (bx + bpd * ((y >> 3) + bpd * (z >> 3))) * kBS3 + kBS * ((y & 7) + kBS * (z & 7));
    }
    __device__ void row(int64_t r, int n, Real (&v)[8]) const
    {
        const Real *p = u + offset_of_row(r, n);
        if constexpr (sizeof(Real) == 4) {
            const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const double2 a = reinterpret_cast<const double2 *>(p)[i];
                v[2 * i] = a.x; v[2 * i + 1] = a.y;
            }
        }
    }
};

constexpr int kLikThreads = 256;  // eight warps: one for each counted term

// The Bernoulli sum of one mask.  A voxel's term depends on its label and, for
// most voxels, on nothing else: where u is above the threshold, and where u -
// uc rounds to -uc (u = 0, or the tumour's far tail), the terms are the same
// four numbers, which are only counted; exp and log1p are left for the
// unlabelled voxels below the threshold in between.
struct Bernoulli {
    double uc, d0;
    int zero[2], above[2];  // by label
    Neumaier rest;
    __device__ void init(double uc_)
    {
        uc = uc_;
        d0 = 0. - uc;
        zero[0] = zero[1] = above[0] = above[1] = 0;
        rest = {0, 0};
    }
    // counts a term that is one of the four; true when it is not
    __device__ __forceinline__ bool count(double d, int label)
    {
        if (d == d0) {
            zero[0] += 1 - label;
            zero[1] += label;
            return false;
        }
        if (d > 0.) {
            above[0] += 1 - label;
            above[1] += label;
            return false;
        }
        return true;
    }
    // the four terms: at u = 0 and above uc (the same for every uc: uc + 1 may
    // round to uc), by label
    static __device__ double term(int which, double uc, double is2)
    {
        double a, b;
        bernoulli_terms(which < 2 ? 0. : 1., which < 2 ? uc : 0., is2, a, b);
        return which & 1 ? a : b;
    }
    // the counted terms added to the sum, each count * term as an exact sum of
    // two doubles
    static __device__ void counted(Neumaier &sum, const long long *n, const double *terms)
    {
        for (int i = 0; i < 4; i++)
            if (n[i]) {
                const double k = (double)n[i], p = k * terms[i];
                sum.add(p);
                sum.add(__fma_rn(k, terms[i], -p));
            }
    }
};
// One voxel of both masks; the exponentials and logarithms of the two side by
// side.
__device__ __forceinline__ void add_voxel(Bernoulli &b1, Bernoulli &b2, double u, int l1, int l2, double is2)
{
    const double lhalf = -0.69314718055994530942;  // log(1/2)
    const double d1 = u - b1.uc, d2 = u - b2.uc;
    const bool q1 = b1.count(d1, l1), q2 = b2.count(d2, l2);
    if (!q1 && !q2) return;
    const double t1 = d1 * d1 * is2, t2 = d2 * d2 * is2;
    double v1 = lhalf - t1, v2 = lhalf - t2;
    if ((q1 && !l1) || (q2 && !l2)) {
        const double e1 = exp(-t1), e2 = exp(-t2);
        const double w1 = log1p(-0.5 * e1), w2 = log1p(-0.5 * e2);
        if (!l1) v1 = w1;
        if (!l2) v2 = w2;
    }
    if (q1) b1.rest.add(d1 < -0.0 ? v1 : lhalf);  // d = 0, and NaN: log(1/2)
    if (q2) b2.rest.add(d2 < -0.0 ? v2 : lhalf);
}
// of one CTA: the PET, T1c and FLAIR sums, the PET voxels and the counts of the
// two masks (zero by label, above by label)
struct LikelihoodPart {
    double sum[6];
    int count[10];
};
static_assert(sizeof(LikelihoodPart) == kLikelihoodPartBytes, "partial size");

// Partial sums of `gridDim.x` CTAs for sample blockIdx.y.  What bounds it: at
// 256^3 with a PET signal the state (4 bytes a voxel in FP32), the masks (2)
// and the PET signal (8) are 235 MB, 36 us at the copy bandwidth; a state whose
// tail covers the brain also takes exp and log1p of most of its voxels, about
// 40 us of FP64.  A thread with its row's eight voxels one by one left half of
// the lanes idle (157 us on a B200), the rows that are not 0 four at a time to
// a warp take 120; before, a dump of the state as doubles, exp and log1p of
// every voxel twice and a final sum by one thread took 830 us.
template <typename State>
__global__ void __launch_bounds__(kLikThreads, 4)
likelihood_partial_kernel(const LikelihoodSample *__restrict__ samples, LikelihoodSample one, int n,
                          const unsigned char *__restrict__ t1c, const unsigned char *__restrict__ flair,
                          const double *__restrict__ pet, const int *__restrict__ roi, int nroi,
                          LikelihoodPart *__restrict__ partial)
{
    constexpr int W = State::kRow;
    const LikelihoodSample &smp = samples ? samples[blockIdx.y] : one;
    const LikelihoodParams p = smp.p;
    const State state = {(decltype(State::u))smp.state};
    const double is2 = 1. / p.slope;
    Neumaier spet = {0, 0};
    int npet = 0;
    Bernoulli b1, b2;
    b1.init(p.t1_uc);
    b2.init(p.t2_uc);
    const int64_t rows = (int64_t)n * n * n / W;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (pet || !roi) {
        for (int64_t r = i0; r < rows; r += stride) {
            typename std::remove_const<typename std::remove_pointer<decltype(State::u)>::type>::type v[W];
            state.row(r, n, v);
            if (!roi) {
                // labels are bytes 0 and 1
                unsigned long long m1, m2;
                if constexpr (W == 8) {
                    m1 = reinterpret_cast<const unsigned long long *>(t1c)[r];
                    m2 = reinterpret_cast<const unsigned long long *>(flair)[r];
                } else {
                    m1 = t1c[r];
                    m2 = flair[r];
                }
                bool any = false;
#pragma unroll
                for (int i = 0; i < W; i++) any |= !(v[i] == 0);
                if (W == 1) {
                    add_voxel(b1, b2, (double)v[0], (int)m1, (int)m2, is2);
                } else {
                    if (!any) {
                        const int k1 = __popcll(m1), k2 = __popcll(m2);
                        b1.zero[0] += W - k1;
                        b1.zero[1] += k1;
                        b2.zero[0] += W - k2;
                        b2.zero[1] += k2;
                    }
                    // the rows that are not 0, four at a time, a voxel per lane
                    // (the rows of a pool are whole warps); their values are in L1
                    const int lane = threadIdx.x & 31, at = state.offset_of_row(r, n);
                    for (unsigned left = __ballot_sync(0xffffffffu, any); left;) {
                        int src = -1;
#pragma unroll
                        for (int g = 0; g < 4; g++) {
                            if (lane >> 3 == g) src = __ffs(left) - 1;
                            left &= left - 1;
                        }
                        const int from = src < 0 ? 0 : src, i = lane & 7;
                        const int o = __shfl_sync(0xffffffffu, at, from);
                        const int l1 = (int)(__shfl_sync(0xffffffffu, m1, from) >> (8 * i)) & 1,
                                  l2 = (int)(__shfl_sync(0xffffffffu, m2, from) >> (8 * i)) & 1;
                        if (src >= 0) add_voxel(b1, b2, (double)state.u[o + i], l1, l2, is2);
                    }
                }
            }
            if (pet) {
                if (p.step_pet != 1) {
                    const int y = (int)(r * W / n % n), z = (int)(r * W / ((int64_t)n * n));
                    if (y % p.step_pet || z % p.step_pet) continue;
                }
                // a row's signal in 16-byte loads, all before the first test (the
                // kernel: 114 us at 256^3 with a signal, 123 with a load per voxel)
                double signal[W];
                if constexpr (W == 8) {
#pragma unroll
                    for (int i = 0; i < W; i += 2) {
                        const double2 q = __ldg(reinterpret_cast<const double2 *>(pet + r * W + i));
                        signal[i] = q.x;
                        signal[i + 1] = q.y;
                    }
                } else signal[0] = pet[r];
                bool on = false;
#pragma unroll
                for (int i = 0; i < W; i++) on |= signal[i] > 0.;
                if (!on) continue;
#pragma unroll
                for (int i = 0; i < W; i++) {
                    const double s = signal[i];
                    if (s > 0. && (p.step_pet == 1 || (int)((r * W + i) % n) % p.step_pet == 0)) {
                        const double d = (double)v[i] - p.pet_scale * s;
                        spet.add(d * d);
                        npet++;
                    }
                }
            }
        }
    }
    if (roi) {
        for (int64_t k = i0; k < nroi; k += stride) {
            const int ix = roi[3 * k], iy = roi[3 * k + 1], iz = roi[3 * k + 2];
            if (ix % p.step_mri != 0 || iy % p.step_mri != 0 || iz % p.step_mri != 0) continue;
            const int64_t g = ix + (int64_t)n * (iy + (int64_t)n * iz);
            add_voxel(b1, b2, state.at(n, ix, iy, iz), t1c[g], flair[g], is2);
        }
    }
    Neumaier v[3] = {spet, b1.rest, b2.rest};
    unsigned k[9] = {(unsigned)npet,        (unsigned)b1.zero[0], (unsigned)b1.zero[1],
                     (unsigned)b1.above[0], (unsigned)b1.above[1], (unsigned)b2.zero[0],
                     (unsigned)b2.zero[1],  (unsigned)b2.above[0], (unsigned)b2.above[1]};
    int total[9];
    __shared__ double red[kLikThreads / 32][6];
    __shared__ unsigned cnt[kLikThreads / 32][9];
    cta_sums(v, k, red, cnt, total);
    if (threadIdx.x != 0) return;
    LikelihoodPart &out = partial[(int64_t)blockIdx.y * gridDim.x + blockIdx.x];
    for (int i = 0; i < 3; i++) {
        out.sum[2 * i] = v[i].s;
        out.sum[2 * i + 1] = v[i].c;
    }
    for (int i = 0; i < 9; i++) out.count[i] = total[i];
}

// The sums of the partials and the four results of sample blockIdx.x, each
// thread over its partials in order (one thread over all of them took 0.15 ms).
__global__ void __launch_bounds__(kLikThreads)
likelihood_final_kernel(const LikelihoodPart *__restrict__ partial, int nparts, int have_pet,
                        const LikelihoodSample *__restrict__ samples, LikelihoodSample one, double *__restrict__ out)
{
    const LikelihoodParams p = (samples ? samples[blockIdx.x] : one).p;
    __shared__ double terms[8];
    const double is2 = 1. / p.slope;
    // the counted terms, by one lane of each warp
    if ((threadIdx.x & 31) == 0) {
        const int w = threadIdx.x >> 5;
        terms[w] = Bernoulli::term(w & 3, w < 4 ? p.t1_uc : p.t2_uc, is2);
    }
    Neumaier v[3] = {};
    unsigned k[9] = {};
    long long total[9];  // a dump grid has up to 2^34 voxels, a warp here at most a seventh of them
    for (int i = threadIdx.x; i < nparts; i += kLikThreads) {
        const LikelihoodPart &q = partial[(int64_t)blockIdx.x * nparts + i];
        for (int j = 0; j < 3; j++) v[j].merge(Neumaier{q.sum[2 * j], q.sum[2 * j + 1]});
        for (int j = 0; j < 9; j++) k[j] += q.count[j];
    }
    __shared__ double red[kLikThreads / 32][6];
    __shared__ unsigned cnt[kLikThreads / 32][9];
    cta_sums(v, k, red, cnt, total);
    if (threadIdx.x != 0) return;
    Bernoulli::counted(v[1], total + 1, terms);
    Bernoulli::counted(v[2], total + 5, terms + 4);
    const double PI = 3.14159265358979323846;
    double lpet = 0;
    if (have_pet) {
        const double p1 = -0.5 * (double)total[0] * log(2. * PI * p.pet_sigma2);
        const double p2 = -0.5 * (1. / p.pet_sigma2) * (v[0].s + v[0].c);
        lpet = p1 + p2;
    }
    out += 4 * (int64_t)blockIdx.x;
    out[0] = lpet;
    out[1] = v[1].s + v[1].c;
    out[2] = v[2].s + v[2].c;
    out[3] = out[0] + out[1] + out[2];
}

// CTAs per sample: enough rows for every thread, at most eight per SM, so
// that the scheduler evens out the CTAs in and outside the tumour (the same for
// one state and for a stage of them, whose results are then the same bits).
int likelihood_parts(int n)
{
    const int64_t rows = (int64_t)n * n * n / 8;
    return (int)std::max<int64_t>(1, std::min<int64_t>(kLikelihoodMaxParts, (rows + kLikThreads - 1) / kLikThreads));
}

namespace {
template <typename State>
cudaError_t launch_likelihood_of(const LikelihoodSample *samples, const LikelihoodSample &one, int count, int n,
                                 const unsigned char *t1c, const unsigned char *flair, const double *pet,
                                 const int *roi, int nroi, void *partial, double *out, cudaStream_t s)
{
    const int parts = likelihood_parts(n);
    LikelihoodPart *part = (LikelihoodPart *)partial;
    likelihood_partial_kernel<State>
        <<<dim3(parts, count), kLikThreads, 0, s>>>(samples, one, n, t1c, flair, pet, roi, nroi, part);
    likelihood_final_kernel<<<count, kLikThreads, 0, s>>>(part, parts, pet != nullptr, samples, one, out);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_likelihood_dense(const double *model, int n, const unsigned char *t1c, const unsigned char *flair,
                                    const double *pet, const int *roi, int nroi, const LikelihoodParams &p,
                                    void *partial, double *out, cudaStream_t s)
{
    return launch_likelihood_of<DenseState>(nullptr, LikelihoodSample{model, p}, 1, n, t1c, flair, pet, roi, nroi,
                                            partial, out, s);
}

template <typename Real>
cudaError_t launch_likelihood_pool(const LikelihoodSample *samples, const LikelihoodSample &one, int count, int n,
                                   const unsigned char *t1c, const unsigned char *flair, const double *pet,
                                   const int *roi, int nroi, void *partial, double *out, cudaStream_t s)
{
    if (n % kBS != 0) return cudaErrorInvalidValue;
    return launch_likelihood_of<PoolState<Real>>(samples, one, count, n, t1c, flair, pet, roi, nroi, partial, out, s);
}

template cudaError_t launch_likelihood_pool<float>(const LikelihoodSample *, const LikelihoodSample &, int, int,
                                                   const unsigned char *, const unsigned char *, const double *,
                                                   const int *, int, void *, double *, cudaStream_t);
template cudaError_t launch_likelihood_pool<double>(const LikelihoodSample *, const LikelihoodSample &, int, int,
                                                    const unsigned char *, const unsigned char *, const double *,
                                                    const int *, int, void *, double *, cudaStream_t);
template cudaError_t launch_uq_dump<float>(const int *, const float *, const float *, int, const float *, int,
                                           double *, cudaStream_t);
template cudaError_t launch_uq_dump<double>(const int *, const double *, const double *, int, const double *, int,
                                            double *, cudaStream_t);

}  // namespace gbfk
