// Runs of RD steps with the blocks resident in shared memory, for uniform
// periodic grids whose blocks sit in consecutive pool slots (any number of
// blocks per direction).  Results are bit-identical to one launch per step
// (rd_step_tma_kernel, rd_step_kernel).
//
// One CTA per SM, launched cooperatively.  Each heavy block (a block with
// tissue in it or its face halos) belongs to one CTA for the whole run: its
// phi (double-buffered), face coefficients and meta words stay in that CTA's
// shared memory, and a step moves only the block's six faces.  A group of
// 128 (or 256) threads steps one block, four (two) x-consecutive cells per
// thread, so that a thread reads its own row, the four neighbouring rows and
// the y and z coefficients in 16-byte (8-byte) accesses.
//
// What bounds it: a step is one exchange of faces through L2 (about 0.9 us
// from a block's stores to the end of its neighbours' next step, what an 8-
// block grid takes) plus the issue of its cells' exact-rounding arithmetic
// (128^3, FP32, 1033 heavy blocks: 1.35 M warp instructions per step, 61 % of
// the issue slots).
// Measured on a B200, us per step over 2000 steps, against one launch per
// step, the seeded brain of 18 % of its box (64^3 182 heavy blocks, 96^3 484,
// 128^3 1033, 160^3 1832): 64^3 FP32 1.13 (3.49), FP64 1.30 (3.86); 96^3 FP32
// 1.30 (9.2, one CTA per block); 128^3 FP32 1.84 (6.36), FP64 2.97 (8.66); 160^3
// FP32 3.15 (17.1, one CTA per block). A stage by teams of CTAs, setup
// included: 128^3 FP32 1.78 us per sample-step (3.2 in launches over all
// samples), 64^3 0.42 (0.96).
//
// Faces travel through L2.  After forming state k a block stores its six
// faces in the exchange buffer k & 1 and its neighbours poll for them there.
// No flag accompanies the data: every value of a clamped state is +0 <= phi
// <= 1 or NaN, so the sign bit of each word is free, and it carries the
// phase (k / 2) & 1 of the buffer's use.  A reader polls until all its words
// show the expected phase.  Two buffers are enough because of the barrier
// between a group's polls and its stores, which every thread of the group takes:
// a group stores state k + 1 of a block only after all its threads have read all
// faces of state k.  So a block that has read its neighbour's state k + 1 knows
// that the neighbour has read its own state k, over which it now stores state
// k + 2.  (The threads that fetch a face are not those that own its cells: a
// barrier of a warp in the place of the group's would let unread words be
// overwritten.)  The phase goes on from launch to launch: the state count lives
// in device memory (index[0]), advanced by the last CTA to leave, so that a
// launch replayed from a graph finds it right too.
//
// Empty blocks (every cell and face-halo cell kEmpty) couple to nothing: all
// face coefficients of a kEmpty cell are exactly 0 (the harmonic mean with a
// zero diffusivity), so with finite values its update is the reaction alone,
// and a heavy block's cell next to an empty block is kEmpty itself.  They
// usually hold +0, which stays; what else they hold, and a NaN, which does
// couple them, is settled after the run (settle_kernel).
#include "gbfk_resident.cuh"

namespace gbfk {
namespace {

// One resident block in shared memory: two states, each with its face halos
// (rows y = -1 .. 8 of planes z = -1 .. 8, and the x faces apart), and the
// face coefficients, in two-value vectors: x faces as eight left faces per row
// and the row's last face apart, y and z faces as in H.  A coefficient carries a set sign bit
// where either cell of the face is kEmpty (see row_cells).
template <typename Real>
struct alignas(16) ResidentBlock {
    ResidentState<Real> st[2];
    Real hx[kBS3], hx8[64], hy[576], hz[576];
    int nbr[6];              // exchange offset (elements) of the face neighbours, -1: an empty block
    int at[6];               // their pool blocks
    int e;                   // block * 4 + block type
    unsigned kinds;          // two bits per warp: the row_cells variant its cells need
};
// All steps of an empty block's cell: no coupling, so the reaction alone
// (cell_rhs with every coefficient +0), until nothing is left of it.
template <typename Real>
__device__ __forceinline__ Real empty_cell_steps(Real phi, int nsteps, Real rho, double dt)
{
#pragma unroll 1
    for (int s = 0; s < nsteps; s++) {
        if (!(phi > (Real)0)) return clamp01(phi);
        const double reaction = __dmul_rn((double)rmul(rho, phi), __dadd_rn(1., -(double)phi));
        phi = cell_update(phi, to_real<Real>(__dadd_rn(0., reaction)), dt);
    }
    return phi;
}

// Whether the empty blocks hold anything but +0 in state 0, noted in `settle` by
// every thread of the grid; other: NULL, or the state buffer that gets them too.
template <typename Real>
__device__ __forceinline__ void scan_empty(const int *empty, int n_empty, const Real *in, Real *other,
                                           SettleWords *settle, unsigned *nan_flag)
{
    const int groups = gridDim.x * (blockDim.x >> 7), g = blockIdx.x * (blockDim.x >> 7) + (threadIdx.x >> 7);
    const int c = (threadIdx.x & 127) * 4;
    bool any = false, bad = false;
    for (int i = g; i < n_empty; i += groups) {
        const int64_t at = (int64_t)empty[i] * kBS3 + c;
        Real v[4];
        ld_cells(in + at, v);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            any |= v[q] != (Real)0;
            bad |= v[q] != v[q];
        }
        if (other) st_cells(other + at, v);
    }
    if (any) settle->outside = 1;
    if (bad) {
        settle->nan = 1;
        atomicOr(nan_flag, 1u);
    }
}

template <typename Real>
__global__ void __launch_bounds__(256) empty_scan_kernel(const int *empty, int n_empty, const Real *in, Real *other,
                                                         SettleWords *settle, unsigned *nan_flag)
{
    scan_empty(empty, n_empty, in, other, settle, nan_flag);
}

// After a run or a chain of steps over the heavy blocks.  With every empty block
// at +0 (every tumour inside the anatomy) and no NaN there is nothing to do, and
// a launch that finds that out costs a call about 3 us.  Else, without a NaN, the
// empty blocks' cells take their steps here, each by itself: a coefficient of 0
// times a finite neighbour is 0.  A NaN does cross such a face into a cell that
// is inside the domain (phi > 0), and stays out of one that is not, which the
// kernels before this one do not tell apart; a NaN stays a NaN, so the last state
// shows that there was one, and all steps of the call are taken again from state
// 0 over all blocks, each cell by the expressions as they are written.
template <typename Real>
__global__ void __launch_bounds__(512, 1) settle_kernel(const __grid_constant__ SettleArgs<Real> a)
{
    constexpr unsigned long long kSettleNs = 10000000000ull;  // the longest any CTA is behind, by far
    __shared__ SettleWords w;
    const int t = threadIdx.x;
    if (t == 0) {
        w.outside = *(volatile unsigned *)&a.words->outside;
        w.nan = *(volatile unsigned *)&a.words->nan;
    }
    __syncthreads();
    if (!w.outside && !w.nan) return;
    const int64_t threads = (int64_t)gridDim.x * blockDim.x, me = (int64_t)blockIdx.x * blockDim.x + t;
    bool bad = false, lost = false, ok = true;
    if (!w.nan) {
        for (int64_t i = me; i < (int64_t)a.n_empty * kBS3; i += threads) {
            Real *p = a.state[a.last] + (int64_t)a.empty[i >> 9] * kBS3 + (i & 511);
            if (*p != (Real)0) *p = empty_cell_steps(*p, a.nsteps, a.rho, a.dt);
        }
    } else {
        Real *here = a.state[0], *there = a.state[1];
        unsigned waits = 0;
        auto grid_sync = [&] {  // false: someone never came
            __threadfence();
            __syncthreads();
            waits++;
            if (t == 0) lost = !arrive_and_wait(a.sync, waits * gridDim.x, kSettleNs);
            return !__syncthreads_or(lost);
        };
        for (int64_t i = me; i < (int64_t)a.n * kBS3; i += threads)
            __stcg(here + (int64_t)(a.items[i >> 9] >> 2) * kBS3 + (i & 511), a.save[i]);
        for (int s = 0; s < a.nsteps && ok; s++) {
            ok = grid_sync();
            for (int64_t i = me; ok && i < (int64_t)a.nblocks * kBS3; i += threads) {
                const int blk = (int)(i >> 9), c = (int)i & 511, x = c & 7, y = (c >> 3) & 7, z = c >> 6;
                const Real phi = __ldcg(here + i);
                Real dphidt = (Real)0.;
                if (in_domain(a.pw[i], a.pg[i], phi)) {
                    auto across = [&](int f, int in) { return (int64_t)block_across(a.bpd, blk, f) * kBS3 + in; };
                    const int64_t at[6] = {x ? i - 1 : across(0, c + 7), x < 7 ? i + 1 : across(1, c - 7),
                                           y ? i - 8 : across(2, c + 56), y < 7 ? i + 8 : across(3, c - 56),
                                           z ? i - 64 : across(4, c + 448), z < 7 ? i + 64 : across(5, c - 448)};
                    Real phn[6];
                    bool low[6];
#pragma unroll
                    for (int k = 0; k < 6; k++) {
                        phn[k] = __ldcg(here + at[k]);
                        low[k] = domain_chf(phn[k], a.pw[at[k]], a.pg[at[k]]) < (Real)0.1;
                    }
                    const Real *h = a.H + (int64_t)blk * kFacesPerBlock;
                    const int rx = (z * 8 + y) * 9 + x, ry = 576 + (z * 9 + y) * 8 + x, rz = 1152 + (z * 8 + y) * 8 + x;
                    dphidt = cell_rhs_flags<Real>(h[rx], h[rx + 1], h[ry], h[ry + 8], h[rz], h[rz + 64], low, phn, phi,
                                                  a.rho, a.ih2);
                }
                const Real next = cell_update(phi, dphidt, a.dt);
                bad |= next != next;
                __stcg(there + i, next);
            }
            Real *const next = here;
            here = there;
            there = next;
        }
        if (ok && here != a.state[a.last]) {
            ok = grid_sync();
            for (int64_t i = me; ok && i < (int64_t)a.nblocks * kBS3; i += threads) __stcg(there + i, __ldcg(here + i));
        }
    }
    if (bad) atomicOr(a.nan_flag, 1u);
    if (!ok && t == 0) atomicOr(a.err_flag, kErrPoll);
    // the last CTA to leave readies the words for the next call
    __syncthreads();
    if (t == 0 && atomicAdd(a.sync + 1, 1u) == gridDim.x - 1) {
        a.sync[0] = a.sync[1] = 0;
        *a.words = SettleWords{};
    }
}

// One run: the blocks of CTA c of G, from state 0 (a.in) to state a.nsteps;
// k0: the states these words of the exchange buffer have carried before (mod
// 4).  False when a face never came (the caller's CTA then leaves).
// The run's arguments lie in constant or shared memory and are read where they
// are used (the waits in between keep the compiler from holding them): with
// 72 registers a thread, what is held spills, and beside 200 KB of blocks the
// spills of 896 threads do not fit in L1 (a 128^3 FP32 stage by teams took 3.7
// us per sample-step with 120 bytes spilled, 2.0 with none).
template <typename Real, int kC, int kGroups, bool kStores>
__device__ __forceinline__ bool run_blocks(const ResidentArgs<Real> &a, double ih2, unsigned long long neg0,
                                           ResidentBlock<Real> *blocks, const int &c, const int &G,
                                           const unsigned &k0)
{
    using TL = Tile<Real, kC, 2>;
    constexpr int kT = kBS3 / kC;  // threads of a group
    constexpr int R = 8 / kC;      // threads of a row
    // skip kStill warps: 128^3 FP32 2.51 -> 2.38 us per step, FP64 3.27 -> 3.11,
    // 64^3 FP64 1.37 -> 1.32; two cells in FP32 lost by it (1.12 -> 1.16)
    constexpr bool kSkips = kC == 4 || sizeof(Real) == 8;
    const int t = threadIdx.x % kT, group = threadIdx.x / kT;
    const int nlocal = a.n > c ? (a.n - 1 - c) / G + 1 : 0;
    const Place w = place_of<Real, kC>(t);
    const int x0 = (t % R) * kC, y = (t / R) & 7, z = t / (8 * R), row = z * 8 + y;
    // the halo vector this thread fetches: kC words of face pf from pw on, to
    // element pd of the state (vectors pstep elements apart); threads beyond
    // the 384 halo cells fetch none
    constexpr bool kAll = kT * kC <= 384;
    const int pf = t * kC / 64, pw = (t * kC) % 64;
    const bool fetches = kAll || pf < 6;
    const int pstep = pf < 2 ? TL::V : kRows * 8 / kC * TL::V;
    const int pd = pf < 2   ? kRows * 8 + pf * 64 + pw
                   : pf < 4 ? TL::template at<kRows>((pw / 8 + 1) * 10 + (pf == 2 ? 0 : 9), pw % 8)
                            : TL::template at<kRows>((pf == 4 ? 0 : 90) + pw / 8 + 1, pw % 8);
    // the faces its own cells belong to: x (one word), y, z (kC words), -1 none
    const int sx = x0 == 0 ? row : x0 + kC == 8 ? 64 + row : -1;
    const int sy = y == 0 ? 128 + z * 8 + x0 : y == 7 ? 192 + z * 8 + x0 : -1;
    const int sz = z == 0 ? 256 + y * 8 + x0 : z == 7 ? 320 + y * 8 + x0 : -1;
    constexpr unsigned kSign = 0x80000000u;
    auto phase_of = [&](unsigned k) { return (k & 2u) ? 0u : kSign; };
    // the faces of a block's state into the exchange buffer
    auto publish = [&](int item, const Real (&v)[kC], unsigned k) {
        Real *ex = a.ex + (((k & 1u) ? a.n : 0) + item) * 384;
        const unsigned m = phase_of(k);
        Real u[kC];
#pragma unroll
        for (int i = 0; i < kC; i++) u[i] = with_phase(v[i], m);
        if (kC == 4 || sx >= 0) st_face1(ex + sx, x0 ? u[kC - 1] : u[0]);
        if (sy >= 0) st_face(ex + sy, u);
        if (sz >= 0) st_face(ex + sz, u);
    };
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kT) : "memory"); };

    group_sync();  // a run before this one has left the group's blocks
    // the group's blocks: state 0, coefficients and cell kinds into shared memory
    for (int j = group; j < nlocal; j += kGroups) {
        ResidentBlock<Real> &b = blocks[j];
        const int item = c + j * G, e = a.items[item];
        const int64_t blk = e >> 2;
        Real p[kC];
        ld_cells(a.in + blk * kBS3 + t * kC, p);
        TL::template store<kRows>(b.st[0].phi, w.tp, p);
        publish(item, p, k0);
        if (a.save) st_cells(a.save + (int64_t)item * kBS3 + t * kC, p);
        if (t == 0) b.e = e;
        if (t < 6) {
            const int nb = a.nbr[item * 6 + t];
            b.nbr[t] = nb < 0 ? -1 : nb * 384;
            b.at[t] = block_across(a.bpd, e >> 2, t);
        }
        if (fetches && a.nbr[item * 6 + pf] < 0) {  // an empty neighbour: +0 for good
            for (int v = 0; v < kC / TL::V; v++)
                for (int i = 0; i < TL::V; i++) b.st[0].phi[pd + v * pstep + i] = b.st[1].phi[pd + v * pstep + i] = (Real)0;
        }
        bool zero = kSkips;
#pragma unroll
        for (int i = 0; i < kC; i++) zero = zero && p[i] == (Real)0;
        load_coefficients<Real, kC>(b, a.H + blk * kFacesPerBlock, a.meta + blk * kBS3, t, zero, group_sync);
    }
    group_sync();

    bool failed = false;
    for (int s = 0; s < a.nsteps; s++) {
        const unsigned k = k0 + s;
        const unsigned m = phase_of(k);
        for (int j = group; j < nlocal; j += kGroups) {
            ResidentBlock<Real> &b = blocks[j];
            ResidentState<Real> &S = b.st[s & 1];
            // the halos of state k: the neighbour across face pf stores its face pf ^ 1
            if (fetches) {
                const int nb = b.nbr[pf];
                if (nb >= 0) {
                    const Real *src = a.ex + (((k & 1u) ? a.n * 384 : 0) + nb + (pf ^ 1) * 64 + pw);
                    Real h[kC];
                    unsigned long long t0 = 0;
                    for (int it = 0;; it++) {
                        ld_face(src, h);
                        unsigned wrong = 0;
#pragma unroll
                        for (int i = 0; i < kC; i++) wrong |= sign_xor(h[i], m);
                        if (!(wrong & kSign)) break;
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
                        Real g[TL::V];
#pragma unroll
                        for (int i = 0; i < TL::V; i++) g[i] = magnitude(h[v * TL::V + i]);
                        st_cells(S.phi + pd + v * pstep, g);
                    }
                }
            }
            // the group's halos are in place, its reads of the state before
            // are over and its writes of state k are seen; a thread that gave
            // up takes its whole group out
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
                return false;
            }
            Real o[kC];
            const unsigned kind = (b.kinds >> (2 * (t >> 5))) & 3u;
            if (kSkips && kind == kStill) {
#pragma unroll
                for (int i = 0; i < kC; i++) o[i] = (Real)0;
            } else {
                Real p[kC];
                TL::template load<kRows>(S.phi, w.tp, p);
                const Real xl = S.phi[w.xl], xr = S.phi[w.xr];
                auto rows = [&](int i, Real (&y0)[2], Real (&y1)[2], Real (&z0)[2], Real (&z1)[2]) {
                    TL::template load2<kRows>(S.phi, w.tp - R, i, y0);
                    TL::template load2<kRows>(S.phi, w.tp + R, i, y1);
                    TL::template load2<kRows>(S.phi, w.tp - 10 * R, i, z0);
                    TL::template load2<kRows>(S.phi, w.tp + 10 * R, i, z1);
                };
                if (kind == kPlain) row_cells<Real, kC, kPlain>(a, ih2, neg0, b, w, p, xl, xr, rows, o);
                else if (kind == kEdge) row_cells<Real, kC, kEdge>(a, ih2, neg0, b, w, p, xl, xr, rows, o);
                else row_cells<Real, kC, kGeneral>(a, ih2, neg0, b, w, p, xl, xr, rows, o);
            }
            if (s + 1 < a.nsteps) {
                publish(c + j * G, o, k + 1);
                TL::template store<kRows>(b.st[(s + 1) & 1].phi, w.tp, o);
            } else {
                bool bad = false;
#pragma unroll
                for (int i = 0; i < kC; i++) bad |= o[i] != o[i];
                if (bad) {  // a NaN stays one: the last state shows it
                    atomicOr(a.nan_flag, 1u);
                    if (a.settle) a.settle->nan = 1;
                }
                if (!kStores || !a.stores) st_cells(a.out + (int64_t)(b.e >> 2) * kBS3 + t * kC, o);
            }
            if (kStores && a.stores) {
                Real *store = a.stores[s];
                if (store) st_cells(store + (int64_t)(b.e >> 2) * kBS3 + t * kC, o);
            }
        }
    }
    return true;
}

template <typename Real, int kC, int kGroups>
__global__ void __launch_bounds__(kGroups * (kBS3 / kC), 1)
resident_run_kernel(const __grid_constant__ ResidentArgs<Real> a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const unsigned k0 = *a.index;  // states stored by earlier launches (mod 4)
    const int c = blockIdx.x, G = gridDim.x;
    run_blocks<Real, kC, kGroups, true>(a, a.ih2, a.neg0, reinterpret_cast<ResidentBlock<Real> *>(smem_raw), c, G, k0);
    if (a.n_empty > 0) scan_empty(a.empty, a.n_empty, a.in, (Real *)nullptr, a.settle, a.nan_flag);
    // the last CTA to leave advances the state count for the next launch
    __syncthreads();
    if (threadIdx.x == 0) {
        if (atomicAdd(a.index + 1, 1u) == gridDim.x - 1) {
            a.index[1] = 0;
            a.index[0] = (k0 + (unsigned)a.nsteps) & 3u;
        }
    }
}

// Many runs at once: team g of the grid's `teams` teams of `size` CTAs takes
// runs off[g] .. off[g + 1], one after the other.  Teams share nothing; a
// run's k0 (start) counts the states its team's exchange buffer carried
// before.
template <typename Real>
struct alignas(16) TeamState {  // at a fixed place in shared memory: no register holds its address
    ResidentArgs<Real> a;
    int run, rank, size, failed;
};
constexpr int kTeamHead = 256;  // bytes of shared memory before the blocks
static_assert(sizeof(TeamState<double>) <= kTeamHead, "team state");
template <typename Real, int kC, int kGroups>
__global__ void __launch_bounds__(kGroups * (kBS3 / kC), 1)
resident_teams_kernel(const ResidentArgs<Real> *runs, const int *off, const int size, double ih2,
                      unsigned long long neg0)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TeamState<Real> &me = *reinterpret_cast<TeamState<Real> *>(smem_raw);
    if (threadIdx.x == 0) {
        me.run = off[blockIdx.x / size];
        me.rank = blockIdx.x % size;
        me.size = size;
        me.failed = 0;
    }
    __syncthreads();
    while (me.run < off[blockIdx.x / size + 1] && !me.failed) {
        // the arguments, word by word
        for (int i = threadIdx.x; i < (int)(sizeof(me.a) / 4); i += blockDim.x)
            reinterpret_cast<unsigned *>(&me.a)[i] = reinterpret_cast<const unsigned *>(runs + me.run)[i];
        __syncthreads();
        if (!run_blocks<Real, kC, kGroups, false>(me.a, ih2, neg0,
                                                  reinterpret_cast<ResidentBlock<Real> *>(smem_raw + kTeamHead),
                                                  me.rank, me.size, me.a.start))
            me.failed = 1;
        __syncthreads();
        if (threadIdx.x == 0) me.run++;
        __syncthreads();
    }
}

// Cells per thread and groups per CTA by the blocks of a CTA (`per`).  Up to
// two blocks the step is a chain of latencies, which two cells per thread
// shorten (64^3 FP32, 2 per CTA: 1.16 us per step against 1.32 with four).
// Beyond, four cells per thread cost fewer instructions. In FP32 a step takes
// about 0.70 us per round of the groups over the blocks and 0.155 us per block
// (the seeded brain scaled to fill every SM: 4 blocks 1.36 us, 6 1.69, 7 1.88, 8
// 2.01, 9 2.57, 12 2.92), so the blocks go in as few rounds as eight groups
// allow (64 registers a thread, none spilled), with no more groups than those
// rounds need (on another brain, 8 blocks: 1.94 us with eight groups, 2.58 with
// seven, 2.38 with four; 9 blocks 2.58 with five, 2.76 with eight; 12 blocks
// 2.94 with six, 3.11 with eight, 3.49 with four). FP64 needs 126 registers for
// four cells: four groups (128^3: 3.07; 3.68 with seven, 4.78 with two cells per
// thread; 4 blocks 1.76, 8 3.19).
constexpr double kRoundUs = 0.70, kBlockUs = 0.155, kRoundUs64 = 1.5;
template <typename Real>
int groups_for(int per, double &us)
{
    if (per <= 2) {
        us = sizeof(Real) == 8 ? 1.33 : 1.15;
        return 2;
    }
    if (sizeof(Real) == 8) {
        us = kRoundUs64 * ((per + 3) / 4);
        return 4;
    }
    const int rounds = (per + 7) / 8, g = (per + rounds - 1) / rounds;
    us = kRoundUs * rounds + kBlockUs * per;
    return g < 4 ? 4 : g;
}
template <typename Real, typename F>
cudaError_t with_shape(int per, F &&f)
{
    using std::integral_constant;
    double us;
    const int g = groups_for<Real>(per, us);
    if (g == 2) return f(integral_constant<int, 2>(), integral_constant<int, 2>());
    if constexpr (sizeof(Real) == 4) {
        if (g == 5) return f(integral_constant<int, 4>(), integral_constant<int, 5>());
        if (g == 6) return f(integral_constant<int, 4>(), integral_constant<int, 6>());
        if (g == 7) return f(integral_constant<int, 4>(), integral_constant<int, 7>());
        if (g == 8) return f(integral_constant<int, 4>(), integral_constant<int, 8>());
    }
    return f(integral_constant<int, 4>(), integral_constant<int, 4>());
}

}  // namespace

void resident_neighbours(int bpd, const int *items, int n, std::vector<int> &nbr)
{
    std::vector<int> at((size_t)bpd * bpd * bpd, -1);
    for (int i = 0; i < n; i++) at[items[i] >> 2] = i;
    for (int i = 0; i < n; i++) {
        const int b = items[i] >> 2;
        const int p[3] = {b % bpd, (b / bpd) % bpd, b / (bpd * bpd)};
        for (int f = 0; f < 6; f++) {
            int q[3] = {p[0], p[1], p[2]};
            q[f >> 1] = (q[f >> 1] + ((f & 1) ? 1 : bpd - 1)) % bpd;
            nbr.push_back(at[q[0] + bpd * (q[1] + bpd * q[2])]);
        }
    }
}

template <typename Real>
int resident_capacity(int sms)
{
    return sms * ((kMaxSmem - kTeamHead) / (int)sizeof(ResidentBlock<Real>));
}

template <typename Real>
double resident_step_us(int per)
{
    double us;
    groups_for<Real>(per, us);
    return us + 0.15;
}

template <typename Real>
cudaError_t launch_resident_run(const ResidentArgs<Real> &a, int sms, cudaStream_t s)
{
    if (a.n <= 0 || a.nsteps <= 0 || a.n > resident_capacity<Real>(sms)) return cudaErrorInvalidValue;
    const int ctas = a.n < sms ? a.n : sms;
    const int per = (a.n + ctas - 1) / ctas;
    return with_shape<Real>(per, [&](auto c, auto g) {
        constexpr int kC = decltype(c)::value, kGroups = decltype(g)::value;
        return launch_coop<resident_run_kernel<Real, kC, kGroups>>(ctas, kGroups * (kBS3 / kC),
                                                                   (size_t)per * sizeof(ResidentBlock<Real>), s, a);
    });
}

template <typename Real>
cudaError_t launch_resident_teams(const ResidentArgs<Real> *runs, const int *off, int teams, int size, int per,
                                  double ih2, cudaStream_t s)
{
    if (teams <= 0 || size <= 0 || per <= 0 || per > resident_capacity<Real>(1))
        return cudaErrorInvalidValue;
    return with_shape<Real>(per, [&](auto c, auto g) {
        constexpr int kC = decltype(c)::value, kGroups = decltype(g)::value;
        return launch_coop<resident_teams_kernel<Real, kC, kGroups>>(
            teams * size, kGroups * (kBS3 / kC), kTeamHead + (size_t)per * sizeof(ResidentBlock<Real>), s, runs, off, size,
            ih2, ResidentArgs<Real>().neg0);
    });
}

template <typename Real>
cudaError_t launch_empty_scan(const int *empty, int n_empty, const Real *in, Real *other, SettleWords *settle,
                              unsigned *nan_flag, cudaStream_t s)
{
    if (n_empty <= 0) return cudaSuccess;
    const int grid = (n_empty + 1) / 2 < 148 * 8 ? (n_empty + 1) / 2 : 148 * 8;
    empty_scan_kernel<Real><<<grid, 256, 0, s>>>(empty, n_empty, in, other, settle, nan_flag);
    return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_settle(const SettleArgs<Real> &a, int sms, cudaStream_t s)
{
    return launch_coop<settle_kernel<Real>>(sms, 512, 0, s, a);
}

template double resident_step_us<float>(int);
template double resident_step_us<double>(int);
template int resident_capacity<float>(int);
template int resident_capacity<double>(int);
template cudaError_t launch_resident_run<float>(const ResidentArgs<float> &, int, cudaStream_t);
template cudaError_t launch_resident_run<double>(const ResidentArgs<double> &, int, cudaStream_t);
template cudaError_t launch_resident_teams<float>(const ResidentArgs<float> *, const int *, int, int, int, double,
                                                  cudaStream_t);
template cudaError_t launch_resident_teams<double>(const ResidentArgs<double> *, const int *, int, int, int, double,
                                                   cudaStream_t);
template cudaError_t launch_empty_scan<float>(const int *, int, const float *, float *, SettleWords *, unsigned *,
                                              cudaStream_t);
template cudaError_t launch_empty_scan<double>(const int *, int, const double *, double *, SettleWords *, unsigned *,
                                               cudaStream_t);
template cudaError_t launch_settle<float>(const SettleArgs<float> &, int, cudaStream_t);
template cudaError_t launch_settle<double>(const SettleArgs<double> &, int, cudaStream_t);

}  // namespace gbfk
