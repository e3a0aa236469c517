// noalloc.cu -- the cell sort of update_neighbors for callers that cannot allocate device memory.
//
// Some hosts give a library no way to allocate GPU memory: an engine that hands out all device
// memory from its own pool, or a plugin that only ever receives buffers from its host.  This
// entry point runs the same counting sort as slf_update_neighbors (cell keys, a count per cell,
// an exclusive scan, ranks by id within each cell) on arrays the caller owns, and keeps its
// scratch in one fixed device array declared at file scope: it never calls cudaMalloc,
// cudaFree or anything that allocates.
//
// The scratch array lives on every GPU that loads this library until the process exits.  It
// caps a call at kNoAllocMaxParticles particles whose bounding box spans at most
// kNoAllocMaxCells cells; larger calls are refused with SLF_ERR_OUT_OF_RANGE.  All calls share
// the array and it keeps what the last call left in it; the kernels clear what must start at
// zero.  Two calls whose work overlaps on the GPU (different streams, or different host threads)
// race on its tables: their orders are wrong, but each has a header of its own (kNoAllocHeaders
// calls in turn), so neither waits for the other's blocks, and no access leaves the array.
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>

#include <cuda_runtime.h>

#include "../../include/solunar_fluid.h"
#include "fluid_device.cuh"
#include "launch.h"
#include "noalloc_grid.h"

namespace slf {

constexpr uint32_t kNoAllocMaxParticles = 1u << 18;  // 262,144 particles
constexpr uint32_t kNoAllocMaxCells = 1u << 20;      // 1,048,576 cells in the bounding box
constexpr uint32_t kNoAllocHeaders = 32;             // headers, taken in turn by the calls
constexpr uint32_t kNoAllocHeader = 2;               // error flag, arrivals (u32 words)

// word offsets inside the scratch array
constexpr size_t kOffBounds = size_t(kNoAllocHeaders) * kNoAllocHeader;  // each block's box (6 words)
constexpr size_t kOffSums = kOffBounds + 6 * kNoAllocBlocks;             // each block's share of the counts
constexpr size_t kOffMembers = kOffSums + kNoAllocBlocks;
constexpr size_t kOffSlots = kOffMembers + kNoAllocMaxParticles;  // where registers do not hold them
constexpr size_t kOffCount = kOffSlots + kNoAllocMaxParticles;
constexpr size_t kNoAllocWords = kOffCount + kNoAllocMaxCells + 1;  // about 6.3 MB

static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocWords];

// header words: error flag, the grid barrier's count of arrivals
enum { kHdrError = 0, kHdrArrived = 1 };
enum { kErrorBox = 1, kErrorWait = 2 };

__device__ __forceinline__ int3 na_cell(const float* pos, uint32_t i, float radius) {
    // cell_of (src/fluid/mod.rs:526-533)
    return make_int3(__float2int_rz(floorf(pos[3 * i] / radius)), __float2int_rz(floorf(pos[3 * i + 1] / radius)),
                     __float2int_rz(floorf(pos[3 * i + 2] / radius)));
}

// All blocks of the grid (a cooperative launch: they are on the GPU together) meet; `round` counts the
// meetings.  A wait ends where a block has left with an error, and one that runs out of patience
// reports itself and lets every block leave.
__device__ __forceinline__ bool na_meet(uint32_t* hdr, uint32_t round) {
    __shared__ bool met;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&hdr[kHdrArrived], 1u);
        const uint32_t all = round * gridDim.x;
        const volatile uint32_t* const seen = hdr;
        bool there = false, left = false;
        for (uint32_t spin = 0; spin < (1u << 22) && !there && !left; ++spin) {
            there = seen[kHdrArrived] >= all;
            if ((spin & 63u) == 63u) left = seen[kHdrError] != 0u;
        }
        if (!there && !left) atomicMax(&hdr[kHdrError], uint32_t(kErrorWait));
        __threadfence();
        met = there;
    }
    __syncthreads();
    return met;
}

// A particle on its way through the passes.
struct NaItem {
    int3 cell;
    uint32_t id, lin, slot, first;
};

// The whole sort in one launch: the box of the cells, a count a cell, their scan, ids by cell, ranks.
// The grid meets between the passes, each pass touches only the box's cells, and a thread's particles
// (their cells, slots and ids) stay in its registers, or, where so few blocks run at once that they do
// not fit there (HELD false), are read again in each pass.  As eight launches over a table of every cell the
// scratch holds, before: 95 -> 60 us a call at 201,544 particles (the call ends with a host wait).  The
// scratch is named here and not passed: with it as a seventh parameter a call took 0.7 us more (30.4 -> 31.1
// at 1,000 particles).
template <bool HELD>
__global__ void __launch_bounds__(kNoAllocThreads) k_na_sort(const float* __restrict__ pos,
                                                             const uint32_t* __restrict__ ids, uint32_t n, float radius,
                                                             uint32_t* hdr, uint32_t* __restrict__ order) {
    uint32_t* const scratch = g_noalloc_scratch;
    uint32_t* const count = scratch + kOffCount;
    uint32_t* const members = scratch + kOffMembers;
    uint32_t* const slots = scratch + kOffSlots;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, width = gridDim.x * kNoAllocThreads;
    __shared__ int part[6][kNoAllocThreads / 32];
    __shared__ uint32_t sums[kNoAllocThreads / 32];
    NaItem held[HELD ? kNoAllocItems : 1];
    // f(item, index) for each of the thread's particles
    auto each = [&](auto&& f) {
        const uint32_t i0 = blockIdx.x * kNoAllocThreads + t;
        if constexpr (HELD) {
#pragma unroll
            for (uint32_t k = 0; k < kNoAllocItems; ++k)
                if (i0 + k * width < n) f(held[k], i0 + k * width);
        } else {
            for (uint32_t i = i0; i < n; i += width) f(held[0], i);
        }
    };
    // (a thread without a particle takes part with an empty box)
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    each([&](NaItem& q, uint32_t i) {
        q.cell = na_cell(pos, i, radius);
        q.id = ids[i];
        lo[0] = min(lo[0], q.cell.x), lo[1] = min(lo[1], q.cell.y), lo[2] = min(lo[2], q.cell.z);
        hi[0] = max(hi[0], q.cell.x), hi[1] = max(hi[1], q.cell.y), hi[2] = max(hi[2], q.cell.z);
    });
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        if (lane == 0) part[a][warp] = lo[a], part[3 + a][warp] = hi[a];
    }
    __syncthreads();
    if (warp < 6) {  // a warp a bound
        const int v = part[warp][lane % (kNoAllocThreads / 32)];
        const int r = warp < 3 ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
        if (lane == 0) scratch[kOffBounds + 6 * blockIdx.x + warp] = uint32_t(r);
    }
    if (!na_meet(hdr, 1)) return;
    // every block takes the box from all blocks' bounds
    __shared__ int box[6];
    if (warp < 6) {
        int v = warp < 3 ? INT_MAX : INT_MIN;
        for (uint32_t b = lane; b < gridDim.x; b += 32) {
            const int w = int(__ldcg(&scratch[kOffBounds + 6 * b + warp]));
            v = warp < 3 ? min(v, w) : max(v, w);
        }
        v = warp < 3 ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
        if (lane == 0) box[warp] = v;
    }
    __syncthreads();
    const long long sx = (long long)box[3] - box[0] + 1, sy = (long long)box[4] - box[1] + 1,
                    sz = (long long)box[5] - box[2] + 1;
    // each side is at most 2^32 cells: bounding them first keeps the products inside 64 bits
    const long long cap = (long long)kNoAllocMaxCells;
    if (sx <= 0 || sy <= 0 || sz <= 0 || sx > cap || sy > cap || sz > cap || sx * sy > cap || sx * sy * sz > cap) {
        if (t == 0) atomicMax(&hdr[kHdrError], uint32_t(kErrorBox));
        return;  // every block alike
    }
    const uint32_t volume = uint32_t(sx * sy * sz);
    for (uint32_t c = blockIdx.x * kNoAllocThreads + t; c < volume; c += width) count[c] = 0u;
    if (!na_meet(hdr, 2)) return;
    // the particle's cell in the table: offsets in 64 bits (a cell minus the box's low corner can pass the
    // i32 range), and every particle checked against the box before it touches the count table: a cell
    // outside it (another call's work on the scratch) fails the call instead of writing outside the array
    auto place = [&](NaItem& q, uint32_t i) {
        if (!HELD) q.cell = na_cell(pos, i, radius);
        const long long x = (long long)q.cell.x - box[0], y = (long long)q.cell.y - box[1],
                        z = (long long)q.cell.z - box[2];
        q.lin = uint32_t((x * sy + y) * sz + z);
        if (x < 0 || x >= sx || y < 0 || y >= sy || z < 0 || z >= sz) {
            atomicMax(&hdr[kHdrError], uint32_t(kErrorBox));
            q.lin = 0u;
        }
    };
    each([&](NaItem& q, uint32_t i) {
        place(q, i);
        q.slot = atomicAdd(&count[q.lin], 1u);
        if (!HELD) slots[i] = q.slot;
    });
    if (!na_meet(hdr, 3)) return;
    // exclusive scan: a run of cells a block, a run of those a thread (whole warps read side by side)
    const uint32_t per = ((volume + gridDim.x - 1) / gridDim.x + 31u) & ~31u;
    const uint32_t c0 = min(blockIdx.x * per, volume), c1 = min(c0 + per, volume);
    uint32_t sum = 0;
    for (uint32_t c = c0 + t; c < c1; c += kNoAllocThreads) sum += __ldcg(&count[c]);
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) sums[warp] = sum;
    __syncthreads();
    if (t == 0) {
        uint32_t all = 0;
        for (int w = 0; w < kNoAllocThreads / 32; ++w) all += sums[w];
        scratch[kOffSums + blockIdx.x] = all;
    }
    if (!na_meet(hdr, 4)) return;
    uint32_t carry = 0;
    for (uint32_t b = lane; b < blockIdx.x; b += 32) carry += __ldcg(&scratch[kOffSums + b]);
    carry = __reduce_add_sync(0xffffffffu, carry);  // (every warp alike)
    for (uint32_t base = c0; base < c1; base += kNoAllocThreads) {
        const uint32_t c = base + t, v = c < c1 ? __ldcg(&count[c]) : 0u;
        uint32_t upto = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t other = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= uint32_t(d)) upto += other;
        }
        __syncthreads();
        if (lane == 31) sums[warp] = upto;
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kNoAllocThreads / 32; ++w) {
            if (uint32_t(w) < warp) before += sums[w];
            all += sums[w];
        }
        if (c < c1) count[c] = carry + before + upto - v;
        carry += all;
    }
    if (blockIdx.x == 0 && t == 0) count[volume] = n;
    if (!na_meet(hdr, 5)) return;
    auto settle = [&](NaItem& q, uint32_t i) {
        if (!HELD) {
            place(q, i);
            q.id = ids[i];
            q.slot = slots[i];  // (this thread wrote it)
        }
        q.first = __ldcg(&count[q.lin]);
    };
    each([&](NaItem& q, uint32_t i) {
        settle(q, i);
        if (q.first < n && q.slot < n - q.first) members[q.first + q.slot] = q.id;
    });
    if (!na_meet(hdr, 6)) return;
    // order[cell start + rank of the id in its cell] = i: the (cell, id) order of mod.rs:541-550.
    // A cell of k particles costs k comparisons a particle (k^2 for the cell).  Equal ids (a world's
    // ids are distinct; a caller's arrays need not be) are ranked by the slot each took in its cell,
    // so order is always a permutation, with repeated ids in no particular order among themselves.
    each([&](NaItem& q, uint32_t i) {
        if (!HELD) settle(q, i);
        const uint32_t e = min(__ldcg(&count[q.lin + 1]), n), own = q.first + q.slot;
        uint32_t rank = 0;
        for (uint32_t k = q.first; k < e; ++k) {
            const uint32_t m = __ldcg(&members[k]);
            rank += (m < q.id || (m == q.id && k < own)) ? 1u : 0u;
        }
        if (q.first < n && rank < n - q.first) order[q.first + rank] = i;
    });
}

namespace {

std::mutex g_noalloc_mutex;
uint32_t* g_noalloc_ptr[256] = {};  // device address of the scratch array, per device ordinal
thread_local uint32_t h_noalloc_error;
std::atomic<uint32_t> g_noalloc_turn{0};

int32_t na_fail(int32_t code, const char* what, cudaError_t e = cudaSuccess) {
    std::string msg = what;
    if (e != cudaSuccess) msg += std::string(": ") + cudaGetErrorString(e);
    set_last_error(msg);
    return code;
}

// The scratch array's device address on the current device, looked up once per device.
int32_t scratch_on_current_device(uint32_t** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return na_fail(SLF_ERR_CUDA, "cudaGetDevice", e);
    if (dev < 0 || dev >= 256) return na_fail(SLF_ERR_CUDA, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return na_fail(SLF_ERR_CUDA, "cudaGetSymbolAddress", e);
        g_noalloc_ptr[dev] = static_cast<uint32_t*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return SLF_OK;
}

// The sort on a grid of at most `room` blocks (0: a block a SM).
int32_t sort_noalloc(const float* positions, const uint32_t* ids, uint64_t n, float radius, uint32_t* order,
                     cudaStream_t s, uint32_t room) {
    if (n == 0) return SLF_OK;
    if (!positions || !ids || !order) return na_fail(SLF_ERR_INVALID_ARGUMENT, "null device pointer");
    if (!(radius > 0.0f) || !std::isfinite(radius)) return na_fail(SLF_ERR_INVALID_ARGUMENT, "radius must be positive");
    if (n > kNoAllocMaxParticles) return na_fail(SLF_ERR_OUT_OF_RANGE, "more particles than the scratch holds");
    uint32_t* scratch = nullptr;
    int32_t st = scratch_on_current_device(&scratch);
    if (st != SLF_OK) return st;
    uint32_t m = uint32_t(n);
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return na_fail(SLF_ERR_CUDA, "cudaDeviceGetAttribute", e);
    const uint32_t all = uint32_t(sms > 0 ? sms : 1);
    room = room && room < all ? room : all;
    uint32_t* hdr = scratch + (g_noalloc_turn.fetch_add(1, std::memory_order_relaxed) % kNoAllocHeaders) * kNoAllocHeader;
    e = cudaMemsetAsync(hdr, 0, kNoAllocHeader * 4, s);
    if (e != cudaSuccess) return na_fail(SLF_ERR_CUDA, "clearing the header", e);
    void* args[] = {&positions, &ids, &m, &radius, &hdr, &order};
    for (;; room /= 2) {
        // (a share of the SMs, of a stream or a process, holds fewer blocks than the device: half as many
        // are tried until they run at once, as one always does)
        const NoAllocGrid grid = noalloc_grid(m, room);
        const void* kernel = grid.held ? reinterpret_cast<const void*>(k_na_sort<true>)
                                       : reinterpret_cast<const void*>(k_na_sort<false>);
        e = cudaLaunchCooperativeKernel(kernel, dim3(grid.blocks), dim3(kNoAllocThreads), args, 0, s);
        if (e != cudaErrorCooperativeLaunchTooLarge || grid.blocks == 1) break;
        cudaGetLastError();
        room = grid.blocks;
    }
    note_launch();
    if (e != cudaSuccess) return na_fail(SLF_ERR_CUDA, "launching the cell sort", e);
    e = cudaMemcpyAsync(&h_noalloc_error, hdr + kHdrError, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return na_fail(SLF_ERR_CUDA, "finishing the cell sort", e);
    if (h_noalloc_error == kErrorWait) return na_fail(SLF_ERR_TIMEOUT, "the cell sort's blocks did not meet");
    if (h_noalloc_error) return na_fail(SLF_ERR_OUT_OF_RANGE, "particles spread over more cells than the scratch holds");
    return SLF_OK;
}

}  // namespace

}  // namespace slf

extern "C" int32_t slf_sort_by_cell_noalloc(const float* positions, const uint32_t* ids, uint64_t n, float radius,
                                            uint32_t* order, void* stream) {
    return slf::sort_noalloc(positions, ids, n, radius, order, static_cast<cudaStream_t>(stream), 0);
}

extern "C" int32_t slf_debug_sort_by_cell_noalloc(const float* positions, const uint32_t* ids, uint64_t n, float radius,
                                                  uint32_t* order, void* stream, uint32_t blocks) {
    return slf::sort_noalloc(positions, ids, n, radius, order, static_cast<cudaStream_t>(stream), blocks);
}
