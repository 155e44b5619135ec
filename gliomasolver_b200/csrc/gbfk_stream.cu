// One RD step of the heavy blocks of a uniform periodic grid that does not fit
// the SMs' shared memory, for calls of several steps (any number of blocks per
// direction).  The empty blocks' steps are made up afterwards (launch_settle):
// nothing couples them to the others while every value is finite, and with a
// NaN all steps are taken again there.  Results are bit-identical to the other
// steps.
//
// A persistent CTA per SM; each group of 128 threads takes blocks of its own,
// four x-consecutive cells per thread, and computes them as the resident runs
// do (row_cells).  What a block needs comes as eight bulk copies that eight
// lanes of the group issue two blocks ahead (one in FP64): the block's cells,
// its six halo faces, and its coefficients as an image laid out once for the
// anatomy and coefficient pair (launch_stream_pack), signs and warp kinds
// included.  So that a halo face is contiguous, every step also writes the x
// and y faces of its blocks apart (z faces are contiguous in the block).  The
// images of a group's first blocks are on their way before the step before has
// finished.
//
// What bounds it, per step: about 4 us from one launch's last block to the next
// one's first (the state cannot be copied before it is complete), then 0.25 us
// (FP32; FP64 0.46) per block of an SM, three quarters of it instruction issue.
// Measured: 256^3 FP32, 7184 heavy blocks, 16.4 us (20.2 with one column of
// cells per thread and tensor boxes as halos, 30 with the empty blocks);
// 216^3 FP32 11.7, 160^3 FP64 8.7, 192^3 FP64 12.7.  Copies by every thread
// (16-, 8- and 4-byte asynchronous ones) took 20.2 at 256^3, their issue queue
// full; six groups 17.1; the sources of the copies through two dependent
// loads instead of a table 20.2.
#include "gbfk_async.cuh"
#include "gbfk_resident.cuh"

namespace gbfk {
namespace {

constexpr int kCells = 4, kThreads = kBS3 / kCells;  // cells of a thread, threads of a group
constexpr unsigned kErrStream = 1u | 1024u;          // error word: a copy never came

template <typename Real>
struct alignas(16) StreamImage {
    Real hx[kBS3], hx8[64], hy[576], hz[576];  // as in ResidentBlock
    int at[6], e;
    unsigned kinds;
};
// x-, x+, y-, y+, z-, z+ halos, as the neighbours' faces: [z][y], [z][x], [y][x]
template <typename Real>
struct alignas(16) StreamSlot {
    Real phi[kBS3], face[6][64];
    StreamImage<Real> b;
};
// Groups per CTA and slots per group: what 227 KB and the registers hold.
template <typename Real>
constexpr int kStreamGroups = sizeof(Real) == 4 ? 7 : 5;
template <typename Real>
constexpr int kStreamSlots = sizeof(Real) == 4 ? 3 : 2;
constexpr int kStreamHead = 256;  // bytes of shared memory for the barriers

// at[block] = its item (the rest: -1)
__global__ void stream_index_kernel(const int *items, int n, int *at)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) at[items[i] >> 2] = i;
}

template <typename Real>
__global__ void __launch_bounds__(kThreads)
stream_pack_kernel(const int *items, int n, int bpd, const Real *H, const unsigned short *meta, const int *at,
                   StreamImage<Real> *image, int *from)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StreamImage<Real> &b = *reinterpret_cast<StreamImage<Real> *>(smem_raw);
    const int t = threadIdx.x, e = items[blockIdx.x];
    const int64_t blk = e >> 2;
    load_coefficients<Real, kCells>(b, H + blk * kFacesPerBlock, meta + blk * kBS3, t, false,
                                    [] { __syncthreads(); });
    if (t == 0) {
        b.e = e;
        from[blockIdx.x * 8] = blockIdx.x;
        from[blockIdx.x * 8 + 1] = (e >> 2) * 8;
    }
    if (t < 6) {
        const int across = block_across(bpd, e >> 2, t), item = at[across];
        b.at[t] = across;
        // in records of 64 cells: x and y faces of the faces array, z faces of
        // the state; an empty neighbour's are the zeros after the last faces
        from[blockIdx.x * 8 + 2 + t] = item < 0 ? (int)(n * 4u | (t < 4 ? 0u : 0x80000000u))
                                       : t < 4  ? item * 4 + (t ^ 1)
                                                : across * 8 + (t == 4 ? 7 : 0);
    }
    __syncthreads();
    const int4 *src = reinterpret_cast<const int4 *>(&b);
    int4 *to = reinterpret_cast<int4 *>(image + blockIdx.x);
    for (int q = t; q < (int)(sizeof(b) / 16); q += kThreads) to[q] = src[q];
}

// The x and y faces of a thread's cells (x0 .. x0 + 3 of row z * 8 + y).
template <typename Real>
__device__ __forceinline__ void put_faces(Real *faces, int t, const Real (&o)[kCells])
{
    const int x0 = (t & 1) * 4, y = (t >> 1) & 7, z = t >> 4;
    faces[(x0 ? 64 : 0) + (t >> 1)] = x0 ? o[3] : o[0];
    if (y == 0 || y == 7) st_cells(faces + (y ? 192 : 128) + z * 8 + x0, o);
}

template <typename Real>
__global__ void __launch_bounds__(kThreads) stream_faces_kernel(const int *items, const Real *phi, Real *faces,
                                                                Real *save)
{
    Real o[kCells];
    ld_cells(phi + (int64_t)(items[blockIdx.x] >> 2) * kBS3 + threadIdx.x * kCells, o);
    put_faces(faces + (int64_t)blockIdx.x * stream_face_values, threadIdx.x, o);
    st_cells(save + (int64_t)blockIdx.x * kBS3 + threadIdx.x * kCells, o);
}

template <typename Real>
__global__ void __launch_bounds__(kStreamGroups<Real> * kThreads, 1)
stream_step_kernel(const __grid_constant__ StreamArgs<Real> a)
{
    constexpr int kG = kStreamGroups<Real>, kSlots = kStreamSlots<Real>, kAhead = kSlots - 1;
    constexpr unsigned kFace = 64 * sizeof(Real);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % kThreads, group = threadIdx.x / kThreads;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw) + group * kSlots;
    StreamSlot<Real> *slots = reinterpret_cast<StreamSlot<Real> *>(smem_raw + kStreamHead) + group * kSlots;
    // this group's blocks: items first, first + stride, ...
    const int first = blockIdx.x + group * gridDim.x, stride = kG * gridDim.x;
    const int mine = a.n > first ? (a.n - 1 - first) / stride + 1 : 0;
    if (t == 0) {
        for (int i = 0; i < kSlots; i++) mbar_init(full + i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    // lane l of the group's first warp copies the image (0), the cells (1) or
    // halo face l - 2; where from, for block i: one load, used a block later
    auto source = [&](int i) { return i < mine ? __ldg(a.from + (first + (int64_t)i * stride) * 8 + t) : 0; };
    auto copy = [&](int i, int from) {
        StreamSlot<Real> &s = slots[i % kSlots];
        uint64_t *bar = full + i % kSlots;
        if (t == 0) bulk_g2s(&s.b, (const StreamImage<Real> *)a.image + from, sizeof(StreamImage<Real>), bar);
        else if (t == 1) bulk_g2s(s.phi, a.in + (int64_t)from * 64, kBS3 * sizeof(Real), bar);
        else {
            const bool apart = t < 6 || from < 0;
            bulk_g2s(s.face[t - 2], (apart ? a.faces_in : a.in) + (int64_t)(from & 0x7fffffff) * 64, kFace, bar);
        }
    };
    constexpr unsigned kBytes = sizeof(StreamImage<Real>) + kBS3 * sizeof(Real) + 6 * kFace;

    // the images and the tables are the call's, the states are the launch before's
    int from[kAhead], next = 0;
    if (t < 8) {
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
            from[i] = source(i);
            if (t == 0 && i < mine) {
                mbar_arrive_expect_tx(full + i, kBytes);
                copy(i, from[i]);
            }
        }
        next = source(kAhead);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (t < 8) {
        __syncwarp(0xffu);
        if (t) {
            asm volatile("fence.proxy.async.global;" ::: "memory");
#pragma unroll
            for (int i = 0; i < kAhead; i++)
                if (i < mine) copy(i, from[i]);
        }
    }
    // the thread's cells and their neighbours, as element offsets in a slot
    const Place w = place_of<Real, kCells>(t);
    const int x0 = (t & 1) * 4, y = (t >> 1) & 7, z = t >> 4, row = t >> 1, c0 = t * kCells;
    const int xl = x0 ? c0 - 1 : kBS3 + row, xr = x0 ? kBS3 + 64 + row : c0 + 4;
    const int ym = y ? c0 - 8 : kBS3 + 128 + z * 8 + x0, yp = y < 7 ? c0 + 8 : kBS3 + 192 + z * 8 + x0;
    const int zm = z ? c0 - 64 : kBS3 + 256 + y * 8 + x0, zp = z < 7 ? c0 + 64 : kBS3 + 320 + y * 8 + x0;
    bool bad = false, lost = false;
    int i = 0;
    for (; i < mine; i++) {
        lost = !mbar_wait(full + i % kSlots, (i / kSlots) & 1);
        // block i is there for everyone, and the slot of block i - 1 is free; a
        // thread that gave up takes its whole group out
        unsigned any;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "barrier.cta.red.or.pred q, %2, %3, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(any)
            : "r"((unsigned)lost), "r"(group + 1), "n"(kThreads)
            : "memory");
        lost = any != 0;
        if (lost) break;
        if (t < 8) {
            if (i + kAhead < mine) {
                if (t == 0) mbar_arrive_expect_tx(full + (i + kAhead) % kSlots, kBytes);
                __syncwarp(0xffu);
                copy(i + kAhead, next);
            }
            next = source(i + kAhead + 1);
        }
        const StreamSlot<Real> &s = slots[i % kSlots];
        const Real *phi = s.phi;
        Real p[kCells], o[kCells];
#pragma unroll
        for (int v = 0; v < 2; v++) {
            Real q[2];
            ld_cells(phi + c0 + 2 * v, q);
            p[2 * v] = q[0];
            p[2 * v + 1] = q[1];
        }
        auto rows = [&](int v, Real (&y0)[2], Real (&y1)[2], Real (&z0)[2], Real (&z1)[2]) {
            ld_cells(phi + ym + 2 * v, y0);
            ld_cells(phi + yp + 2 * v, y1);
            ld_cells(phi + zm + 2 * v, z0);
            ld_cells(phi + zp + 2 * v, z1);
        };
        const unsigned kind = (s.b.kinds >> (2 * (t >> 5))) & 3u;
        if (kind == kPlain) row_cells<Real, kCells, kPlain>(a, a.ih2, a.neg0, s.b, w, p, phi[xl], phi[xr], rows, o);
        else if (kind == kEdge) row_cells<Real, kCells, kEdge>(a, a.ih2, a.neg0, s.b, w, p, phi[xl], phi[xr], rows, o);
        else row_cells<Real, kCells, kGeneral>(a, a.ih2, a.neg0, s.b, w, p, phi[xl], phi[xr], rows, o);
        st_cells(a.out + (int64_t)(s.b.e >> 2) * kBS3 + c0, o);
        put_faces(a.faces_out + (first + (int64_t)i * stride) * stream_face_values, t, o);
#pragma unroll
        for (int q = 0; q < kCells; q++) bad |= o[q] != o[q];
    }
    if (bad) {
        atomicOr(a.nan_flag, 1u);
        a.settle->nan = 1;
    }
    if (lost && t == 0) {
        atomicOr(a.err_flag, kErrStream);
        // the copies in flight land before the CTA's shared memory goes away
        for (int j = i; j < mine && j < i + kAhead; j++) mbar_wait(full + j % kSlots, (j / kSlots) & 1);
    }
}

}  // namespace

template <typename Real>
size_t stream_image_bytes() { return sizeof(StreamImage<Real>); }

template <typename Real>
cudaError_t launch_stream_pack(const int *items, int n, int bpd, const Real *H, const unsigned short *meta,
                               void *image, int *from, int *at, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(at, 0xff, (size_t)bpd * bpd * bpd * sizeof(int), s);
    if (e != cudaSuccess) return e;
    stream_index_kernel<<<(n + 255) / 256, 256, 0, s>>>(items, n, at);
    stream_pack_kernel<Real><<<n, kThreads, sizeof(StreamImage<Real>), s>>>(items, n, bpd, H, meta, at,
                                                                            (StreamImage<Real> *)image, from);
    return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_stream_faces(const int *items, int n, const Real *phi, Real *faces, Real *save, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    stream_faces_kernel<Real><<<n, kThreads, 0, s>>>(items, phi, faces, save);
    return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_stream_step(const StreamArgs<Real> &a, bool first, int sms, cudaStream_t s)
{
    if (a.n <= 0) return cudaSuccess;
    constexpr int kG = kStreamGroups<Real>;
    constexpr size_t smem = kStreamHead + sizeof(StreamSlot<Real>) * kStreamSlots<Real> * kG;
    static_assert(smem <= kMaxSmem && kStreamSlots<Real> * kG * 8 <= kStreamHead, "slots");
    cudaError_t e = raise_smem<stream_step_kernel<Real>>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n < sms ? a.n : sms);
    cfg.blockDim = dim3(kG * kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = first ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, stream_step_kernel<Real>, a);
}

template size_t stream_image_bytes<float>();
template size_t stream_image_bytes<double>();
template cudaError_t launch_stream_pack<float>(const int *, int, int, const float *, const unsigned short *, void *,
                                               int *, int *, cudaStream_t);
template cudaError_t launch_stream_pack<double>(const int *, int, int, const double *, const unsigned short *, void *,
                                               int *, int *, cudaStream_t);
template cudaError_t launch_stream_faces<float>(const int *, int, const float *, float *, float *, cudaStream_t);
template cudaError_t launch_stream_faces<double>(const int *, int, const double *, double *, double *, cudaStream_t);
template cudaError_t launch_stream_step<float>(const StreamArgs<float> &, bool, int, cudaStream_t);
template cudaError_t launch_stream_step<double>(const StreamArgs<double> &, bool, int, cudaStream_t);

}  // namespace gbfk
