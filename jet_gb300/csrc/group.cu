// Grouped launch of small contractions: several independent (batched)
// products C[b] = A[b] B[b] in one kernel.
//
// The reference runs every path step as its own ContractTensors call
// (Tensor.hpp:708-752: two transposes, then one BLAS call). For the many small
// slice-dependent steps of a sliced network that is one to three launches per
// step, each too small to fill the GPU. Here a run of such steps that do not
// read each other's outputs goes into one launch.
// Each operand is read through offset tables instead of a transpose pass:
// element (b, i, j) of the product's view of A is A[a_bat[b] + a_row[i] +
// a_col[j]], so any permutation of the operand's axes and any placement of
// the batch axes is absorbed into the load. C is written packed, batch x m x
// n, row-major, as jetgpu_contract_batched writes it.
//
// CTA tiles are 32 x 32 outputs of one (task, batch item), 256 threads, FP32
// or FP64 FMAs over k in order (the plain form's arithmetic).
//
// Bound by latency: the tasks of a circuit network are a few outputs over a
// few k (2 x 2 x 8), and a level's launch is a chain of dependent loads (task,
// offset tables, elements). A tile of little work (kFlatWork) gives one output
// to each thread, which reads its k values straight through the tables with
// all loads of eight k issued before any arithmetic: no staging, no barrier.
// Through staged 32 x 32 x 32 slices, mostly padding, the smallest launch took
// 7.5 us. Tiles of more work are staged in shared memory, 2 x 2 outputs a
// thread. Whole k in one stage (64 of complex64) measured the same.
// The launch uses programmatic stream serialisation, so that a chain of levels
// overlaps each launch with the end of the one before. Where the tables were
// uploaded by a copy (`uploaded`: the executors' launches), a launch reads them
// -- tile scan, task, offsets: three of its five dependent loads -- before it
// waits. 16-qubit amplitude replay (13 levels) 124 -> 103 us, 720-angle gradient
// (53 launches) 1,455 -> 1,375 us, 81 qutrit slices 4,494 -> 4,409 us (without any
// early start 1,477 and 4,498). Tables that a kernel may have just written are
// read after the wait.
//  * What a launch may read before its wait: these launches and skinny.cu's tiny
//    steps let the next one start before they wait themselves, so in an unbroken
//    run of them a launch may start while any earlier one of the run, and the
//    kernel that the run follows, still execute. Its tables must have been
//    complete when that kernel started: copied before it, or directly before the
//    run (a launch starts early behind a kernel only), or waited for by the host,
//    as the executors do once after they upload theirs.
//  * The wait ends when the launch before has ended, which waited for the one
//    before it: everything earlier has ended too, and its writes are visible.
//  * What an earlier launch of the run may write (operands; task arrays that were
//    not uploaded) is read by plain loads: no pointer to it is const
//    __restrict__, whose loads may take the non-coherent path, which is for memory
//    that nobody writes while the kernel runs.
#include "common.cuh"

namespace jetgpu {
namespace {

constexpr int kGT = 32;       // output tile edge
constexpr int kGK = 32;       // k slice
constexpr int kMaxTasks = 256; // tasks per launch
constexpr int kGThreads = 256; // threads per CTA: one per task in the tile prefix scan
static_assert(kGThreads == kMaxTasks, "the prefix scan reads one task per thread");

template <typename T> struct V2;
template <> struct V2<float> {
    using type = float2;
};
template <> struct V2<double> {
    using type = double2;
};

// Most multiply-adds of a tile that goes through the tables directly (8 k of a
// full 32 x 32 tile), and its longest k.
// And its most outputs: with 4 a thread, complex64 is slower than staged (one
// 32 x 32 x 2..8 task 5.4 us, staged 5.0; 6 of 256 x 256 x 1 8.4 and 7.9), where
// complex128, whose padding costs FP64 adds, takes 12 us and staged 36.
constexpr uint64_t kFlatWork = 8192;
constexpr uint64_t kFlatK = 64;
template <typename T> constexpr uint32_t kFlatOutputs = sizeof(T) == 4 ? 512 : 1024;

template <typename V> __device__ __forceinline__ void GroupMac(V &acc, const V &a, const V &b)
{
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
}

template <typename T, bool kUploaded>
__device__ __forceinline__ void GroupContract(const jetgpu_group_task *tasks, int n_tasks,
                                              uint64_t total_tiles)
{
    using V = typename V2<T>::type;
    __shared__ uint64_t first_tile[kMaxTasks + 1];
    __shared__ uint64_t warp_sum[kGThreads / 32];
    __shared__ V As[kGK][kGT + 1];
    __shared__ V Bs[kGK][kGT + 1];
    // The wait for the kernel before: at the latest before the first operand.
    bool waited = false;
    const auto wait = [&]() {
        if (!waited)
            asm volatile("griddepcontrol.wait;" ::: "memory");
        waited = true;
    };
    if (!kUploaded)
        wait();
    // The next launch may start once every CTA is past this.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // First tile of every task: thread t reads task t's tile count, then an
    // inclusive scan by warps and over the eight warp sums.
    {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        uint64_t sum = 0;
        if (tid < n_tasks) {
            const jetgpu_group_task &q = tasks[tid];
            sum = q.batch * ((q.m + kGT - 1) / kGT) * ((q.n + kGT - 1) / kGT);
        }
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint64_t add = __shfl_up_sync(0xffffffffu, sum, off);
            if (lane >= off)
                sum += add;
        }
        if (lane == 31)
            warp_sum[warp] = sum;
        __syncthreads();
        for (int w = 0; w < warp; ++w)
            sum += warp_sum[w];
        first_tile[tid + 1] = sum;
        if (tid == 0)
            first_tile[0] = 0;
        __syncthreads();
    }
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16; // 2 x 2 outputs each
    for (uint64_t g = blockIdx.x; g < total_tiles; g += gridDim.x) {
        // The last task whose first tile is at most g.
        int t = 0;
#pragma unroll
        for (int step = kMaxTasks / 2; step > 0; step >>= 1)
            if (t + step < n_tasks && first_tile[t + step] <= g)
                t += step;
        const jetgpu_group_task *task = tasks + t;
        if constexpr (!kUploaded) {
            // Its own copy: read by plain loads, the fields would be read again
            // after every store.
            __shared__ jetgpu_group_task copy;
            constexpr int kWords = sizeof(jetgpu_group_task) / sizeof(uint64_t);
            __syncthreads(); // the tile before has been read
            if (threadIdx.x < kWords)
                reinterpret_cast<uint64_t *>(&copy)[threadIdx.x] =
                    reinterpret_cast<const uint64_t *>(task)[threadIdx.x];
            __syncthreads();
            task = &copy;
        }
        const jetgpu_group_task &q = *task;
        const uint64_t local = g - first_tile[t];
        const uint64_t tiles_n = (q.n + kGT - 1) / kGT;
        const uint64_t tiles_mn = ((q.m + kGT - 1) / kGT) * tiles_n;
        const uint64_t b = local / tiles_mn;
        const uint64_t r = local - b * tiles_mn;
        const uint64_t m0 = (r / tiles_n) * kGT, n0 = (r % tiles_n) * kGT;
        const V *A = static_cast<const V *>(q.A) + q.a_bat[b];
        const V *B = static_cast<const V *>(q.B) + q.b_bat[b];
        V *C = static_cast<V *>(q.C) + b * q.m * q.n;
        const uint32_t rows = (uint32_t)min(q.m - m0, (uint64_t)kGT);
        const uint32_t cols = (uint32_t)min(q.n - n0, (uint64_t)kGT);
        if (q.k <= kFlatK && rows * cols <= kFlatOutputs<T> && rows * cols * q.k <= kFlatWork) {
            const uint32_t k = (uint32_t)q.k;
            for (uint32_t e = threadIdx.x; e < rows * cols; e += kGThreads) {
                const uint32_t i = e / cols, j = e - i * cols;
                const V *pa = A + q.a_row[m0 + i];
                const V *pb = B + q.b_col[n0 + j];
                V acc{0, 0};
                for (uint32_t k0 = 0; k0 < k; k0 += 8) {
                    uint64_t ao[8], bo[8];
                    V av[8], bv[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) { // past k: the last product's loads again
                        const uint32_t kk = min(k0 + u, k - 1);
                        ao[u] = q.a_col[kk];
                        bo[u] = q.b_row[kk];
                    }
                    wait();
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        av[u] = pa[ao[u]];
                        bv[u] = pb[bo[u]];
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (k0 + u < k)
                            GroupMac(acc, av[u], bv[u]);
                }
                wait(); // no k: nothing was read
                C[(m0 + i) * q.n + n0 + j] = acc;
            }
            continue;
        }
        V acc[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                acc[i][j] = V{0, 0};
        for (uint64_t k0 = 0; k0 < q.k; k0 += kGK) {
            // 32 x 32 of A (rows m0.., k k0..) and of B (k k0.., cols n0..):
            // 4 elements of each per thread, consecutive threads along k for A
            // and along n for B.
            uint64_t ao[4], bo[4];
            bool av[4], bv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int idx = threadIdx.x + 256 * e;
                const int rr = idx / kGK, cc = idx % kGK;
                const uint64_t gi = m0 + rr, gk = k0 + cc;
                av[e] = gi < q.m && gk < q.k;
                ao[e] = av[e] ? q.a_row[gi] + q.a_col[gk] : 0;
                const uint64_t gk2 = k0 + rr, gj = n0 + cc;
                bv[e] = gk2 < q.k && gj < q.n;
                bo[e] = bv[e] ? q.b_row[gk2] + q.b_col[gj] : 0;
            }
            wait();
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int idx = threadIdx.x + 256 * e;
                const int rr = idx / kGK, cc = idx % kGK;
                As[cc][rr] = av[e] ? A[ao[e]] : V{0, 0};
                Bs[rr][cc] = bv[e] ? B[bo[e]] : V{0, 0};
            }
            __syncthreads();
#pragma unroll 8
            for (int kk = 0; kk < kGK; ++kk) {
                const V a0 = As[kk][ty], a1 = As[kk][ty + 16];
                const V b0 = Bs[kk][tx], b1 = Bs[kk][tx + 16];
                const V av[2] = {a0, a1}, bv[2] = {b0, b1};
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        GroupMac(acc[i][j], av[i], bv[j]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint64_t gi = m0 + ty + 16 * i, gj = n0 + tx + 16 * j;
                if (gi < q.m && gj < q.n)
                    C[gi * q.n + gj] = acc[i][j];
            }
    }
    wait(); // a launch never ends before the one that it started behind
}

// The task array may be the output of the kernel before.
template <typename T>
__global__ void __launch_bounds__(kGThreads)
    group_contract_kernel(const jetgpu_group_task *tasks, int n_tasks, uint64_t total_tiles)
{
    GroupContract<T, false>(tasks, n_tasks, total_tiles);
}

// The task array is complete: its fields are read again where they are used (64
// registers in complex64; kept, 94).
template <typename T>
__global__ void __launch_bounds__(kGThreads)
    group_uploaded_kernel(const jetgpu_group_task *__restrict__ tasks, int n_tasks,
                          uint64_t total_tiles)
{
    GroupContract<T, true>(tasks, n_tasks, total_tiles);
}

int LaunchGroup(const jetgpu_group_task *tasks, int n_tasks, uint64_t total_tiles, int dtype,
                void *stream, bool uploaded)
{
    NvtxRange range("jetgpu_contract_group");
    ClearError();
    JETGPU_REQUIRE(dtype == JETGPU_C64 || dtype == JETGPU_C128, "bad dtype");
    JETGPU_REQUIRE(n_tasks >= 0 && n_tasks <= kMaxTasks, "at most 256 tasks per group");
    if (n_tasks == 0 || total_tiles == 0)
        return JETGPU_OK;
    JETGPU_REQUIRE(tasks != nullptr, "null task table");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(GridFor(total_tiles, 8));
    cfg.blockDim = dim3(kGThreads);
    cfg.stream = AsStream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    JETGPU_CUDA_TRY(cudaLaunchKernelEx(
        &cfg,
        dtype == JETGPU_C64
            ? (uploaded ? group_uploaded_kernel<float> : group_contract_kernel<float>)
            : (uploaded ? group_uploaded_kernel<double> : group_contract_kernel<double>),
        tasks, n_tasks, total_tiles));
    return CheckLaunch(uploaded ? "group_uploaded_kernel" : "group_contract_kernel");
}

} // namespace
} // namespace jetgpu

using namespace jetgpu;

extern "C" {

uint64_t jetgpu_group_tiles(uint64_t batch, uint64_t m, uint64_t n)
{
    return batch * ((m + kGT - 1) / kGT) * ((n + kGT - 1) / kGT);
}

int jetgpu_contract_group(const jetgpu_group_task *tasks, int n_tasks, uint64_t total_tiles,
                          int dtype, void *stream)
{
    return LaunchGroup(tasks, n_tasks, total_tiles, dtype, stream, false);
}

int jetgpu_contract_group_uploaded(const jetgpu_group_task *tasks, int n_tasks,
                                   uint64_t total_tiles, int dtype, void *stream)
{
    return LaunchGroup(tasks, n_tasks, total_tiles, dtype, stream, true);
}

} // extern "C"
