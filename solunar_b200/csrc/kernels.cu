// kernels.cu -- the fluid substep on the device.
//
// One thread per particle, or, in small scenes' density and WCSPH force passes, several lanes of a warp.
// Particles live in SoA float4 arrays (x, y, z and what a pass leaves for the gathers of the next: p / rho^2
// or the stiffness beside a position, the density beside a velocity, PairRecords),
// sorted by (cell, id) like the reference's arrays (src/fluid/mod.rs:540-566); every pass reads
// neighbours through the cell tables in the reference's list order, so each particle's sums are
// the reference's sequential sums, bit for bit.  Grid-wide reductions (bounding box, fastest
// particle, solver residual) are block trees feeding one atomic or one last-block finish per
// launch; the residual is summed in double-double (compensated), deterministically.
#include <atomic>
#include <cfloat>
#include <climits>
#include <type_traits>

#include "fluid_device.cuh"
#include "launch.h"
#include "reduce.cuh"
#include "scan.cuh"

namespace slf {

// Bounding box of cells, fastest speed, held-back count and non-finite flag of a block's
// particles, folded into the status with one atomic each (a thread without particles: an empty box).
__device__ __forceinline__ void fold_advance_box(Status* st, int3 lo, int3 hi, float speed, uint32_t held,
                                                 uint32_t bad) {
    uint32_t sb = speed > 0.0f ? __float_as_uint(speed) : 0u;
    int lox = block_reduce(lo.x, MinI(), INT_MAX);
    int loy = block_reduce(lo.y, MinI(), INT_MAX);
    int loz = block_reduce(lo.z, MinI(), INT_MAX);
    int hix = block_reduce(hi.x, MaxI(), INT_MIN);
    int hiy = block_reduce(hi.y, MaxI(), INT_MIN);
    int hiz = block_reduce(hi.z, MaxI(), INT_MIN);
    sb = block_reduce(sb, MaxU(), 0u);
    held = block_reduce(held, SumU(), 0u);
    bad = block_reduce(bad, MaxU(), 0u);
    if (threadIdx.x == 0) {
        if (lox != INT_MAX) {
            atomicMin(&st->cell_lo[0], lox);
            atomicMin(&st->cell_lo[1], loy);
            atomicMin(&st->cell_lo[2], loz);
            atomicMax(&st->cell_hi[0], hix);
            atomicMax(&st->cell_hi[1], hiy);
            atomicMax(&st->cell_hi[2], hiz);
        }
        if (sb) atomicMax(&st->vmax_bits, sb);
        if (held) atomicAdd(&st->held, held);
        if (bad) atomicMax(&st->nonfinite, 1u);
    }
}

// The same with one particle a thread (valid: whether it has one).
__device__ __forceinline__ void fold_advance_stats(Status* st, bool valid, int3 c, float speed, uint32_t held,
                                                   uint32_t bad) {
    const int3 lo = make_int3(INT_MAX, INT_MAX, INT_MAX), hi = make_int3(INT_MIN, INT_MIN, INT_MIN);
    fold_advance_box(st, valid ? c : lo, valid ? c : hi, valid ? speed : 0.0f, held, bad);
}

// ---- bounding box and fastest speed of the current state ---------------------------------

__global__ void k_state_stats(Params p, const float4* __restrict__ pos, const float4* __restrict__ vel,
                              Status* st) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = i < p.n;
    int3 c = make_int3(0, 0, 0);
    float speed = 0.0f;
    if (valid) {
        float4 a = pos[i];
        float4 v = vel[i];
        c = cell_of(p, a.x, a.y, a.z);
        // Vec3::length (step.rs:92-96)
        speed = sqrtf(dot3(v.x, v.y, v.z, v.x, v.y, v.z));
        if (!(speed == speed)) speed = 0.0f;  // f32::max ignores NaN
    }
    fold_advance_stats(st, valid, c, speed, 0u, 0u);
}

// max(0, rho / rest - 1) over the particles (step.rs:84-88)
__global__ void k_max_compression(Params p, const float* __restrict__ rho, Status* st) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t b = 0;
    if (i < p.n) {
        float c = rho[i] / p.rest - 1.0f;
        if (c > 0.0f) b = __float_as_uint(c);
    }
    b = block_reduce(b, MaxU(), 0u);
    if (threadIdx.x == 0 && b) atomicMax(&st->maxcomp_bits, b);
}

// The status into the host's pinned copy, then the word the host polls.  A copy and a stream
// synchronisation in its place take about 6 us more a wait: 44 -> 38 us a substep of 720 particles.
// spoiled (optional): whether the substep's lists outgrew cap or its values are non-finite.
__global__ void __launch_bounds__(32) k_post_status(const Status* st, Status* out, uint32_t* posted, uint32_t cap,
                                                    uint32_t* spoiled) {
    constexpr uint32_t words = sizeof(Status) / 4;
    static_assert(sizeof(Status) % 4 == 0 && words <= 32, "a word a lane");
    const uint32_t t = threadIdx.x;
    if (t < words)
        reinterpret_cast<volatile uint32_t*>(out)[t] = reinterpret_cast<const volatile uint32_t*>(st)[t];
    if (t == 0 && spoiled) *spoiled = st->list_max > cap || st->nonfinite ? 1u : 0u;
    __threadfence_system();
    __syncwarp();
    if (t == 0) *reinterpret_cast<volatile uint32_t*>(posted) = 1u;
}

// ---- spatial hash: counting sort by dense cell index, then id within each cell ------------

// cells (cell-relative positions) non-null: the cell is stored, not computed
// begin (a substep recorded as a graph, or a WCSPH substep launch by launch): the status starts afresh,
// and the substep's constants come from the host's copy, which it writes before each launch
__global__ void k_count_cells(Params p, const float4* __restrict__ pos, const int4* __restrict__ cells, int3 low,
                              int3 span, uint32_t* count, uint32_t* lin, uint32_t* slot, SubstepBegin begin) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (begin.status && i == 0) {
        Status z{};
        z.cell_lo[0] = z.cell_lo[1] = z.cell_lo[2] = INT_MAX;
        z.cell_hi[0] = z.cell_hi[1] = z.cell_hi[2] = INT_MIN;
        *begin.status = z;
        *begin.consts = *begin.from;
    }
    uint32_t l = 0xffffffffu;  // (no cell: tables hold fewer than 2^31)
    if (i < p.n) {
        int3 c;
        if (cells) {
            int4 c4 = cells[i];
            c = make_int3(c4.x, c4.y, c4.z);
        } else {
            float4 a = pos[i];
            c = cell_of(p, a.x, a.y, a.z);
        }
        long long x = (long long)c.x - low.x, y = (long long)c.y - low.y, z = (long long)c.z - low.z;
        // the box was taken over these very positions; stay in bounds regardless
        x = x < 0 ? 0 : (x >= span.x ? span.x - 1 : x);
        y = y < 0 ? 0 : (y >= span.y ? span.y - 1 : y);
        z = z < 0 ? 0 : (z >= span.z ? span.z - 1 : z);
        l = (uint32_t)((x * span.y + y) * span.z + z);
        lin[i] = l;
    }
    // One atomic for a run of the warp's particles in one cell: a running state is about sorted, and one
    // that is not pays a shuffle and a ballot.  Against an atomic a particle, us, sorted / shuffled: 250k
    // of support 4 (64 to a cell) 15.1 -> 8.0 / 12.9 -> 13.4, 1M of support 2 11.9 -> 12.2 / 17.4 -> 17.7
    // (with the warp's particles of a cell matched wherever they stand: 8.3 / 13.5, 12.4 / 29.3).
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t left = __shfl_up_sync(0xffffffffu, l, 1);
    const bool head = lane == 0u || left != l;
    const uint32_t heads = __ballot_sync(0xffffffffu, head);
    const uint32_t upto = 0xffffffffu >> (31u - lane);  // this lane and those before it
    const uint32_t after = heads & ~upto;
    uint32_t at = 0;
    if (head && i < p.n) at = atomicAdd(&count[l], (after ? uint32_t(__ffs(int(after))) - 1u : 32u) - lane);
    const uint32_t first = 31u - uint32_t(__clz(int(heads & upto)));
    at = __shfl_sync(0xffffffffu, at, int(first));
    if (i < p.n) slot[i] = at + lane - first;
}

// GridDev::near of a dense table, a thread a cell
__global__ void k_grid_near(GridDev g, uint32_t* __restrict__ near) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= uint32_t(g.sx) * uint32_t(g.sy) * uint32_t(g.sz)) return;
    const int z = int(c % uint32_t(g.sz)), y = int(c / uint32_t(g.sz) % uint32_t(g.sy)),
              x = int(c / uint32_t(g.sz) / uint32_t(g.sy));
    uint32_t mask = 0;
    for (int t = 0; t < 27; ++t) {
        const int qx = x + t % 3 - 1, qy = y + t / 3 % 3 - 1, qz = z + t / 9 - 1;
        if (qx < 0 || qx >= g.sx || qy < 0 || qy >= g.sy || qz < 0 || qz >= g.sz) continue;
        const uint32_t q = (uint32_t(qx) * uint32_t(g.sy) + uint32_t(qy)) * uint32_t(g.sz) + uint32_t(qz);
        if (__ldg(&g.start[q + 1]) > __ldg(&g.start[q])) mask |= 1u << t;
    }
    near[c] = mask;
}

__global__ void k_scatter_members(uint32_t n, const uint32_t* __restrict__ lin, const uint32_t* __restrict__ slot,
                                  const uint32_t* __restrict__ start, const uint32_t* __restrict__ ids,
                                  uint32_t* members) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    members[start[lin[i]] + slot[i]] = ids[i];
}

// ---- the walk order of the list passes (PairLists::order) -------------------------------------
// Cells taken in 2 x 2-column bricks whose z is split in quads, key = ((x / 2, y / 2), z / 4, x % 2,
// y % 2, z % 4): 256 consecutive rows cover about 2 x 2 x 8 cells instead of a 1 x 1 x 32 column,
// and a warp's 32 rows are (about) four consecutive cells of one column, whose neighbours lie in
// consecutive cells of the same neighbouring columns.
//
// The row of cell (x, y, z)'s first member needs no scan over the keys: the particles are sorted
// x-major, so the members of any run of cells along z, or of a run of columns along y, are one
// difference of the cell table.  Before the cell come the slab pairs before its own, the bricks
// before its own in the slab pair, the quads before its own in the four columns, the columns
// before its own in the quad, and the cells before it in its column.  A dozen loads from the table's
// cache lines in k_rank_reorder (17 -> 21 us at 1M) in place of a count, a scan and a fill of the
// keys (six nodes, 30 us at 1M and 26 at 75k).
// Bricks begin at the box's own corner, not at the padding's: a cell further out, they split the pairs and
// quads that water against a container fills (us with the bricks on the padding and on the corner: EXACT
// density 435 -> 415 at 1M and 247 -> 231 at 500k, check 69 -> 67 at 500k; FAST push of 8,000 particles at
// support 4 63.9 -> 61.8).  Over 36 shapes of 8k to 600k particles the passes take 0.6 % less in sum, single
// shapes up to 4 % more or 7 % less.
__device__ __forceinline__ uint32_t walk_row(const uint32_t* __restrict__ start, int3 span, int pad, uint32_t lin) {
    const uint32_t sy = uint32_t(span.y), sz = uint32_t(span.z);
    const int z = int(lin % sz), y = int(lin / sz % sy), x = int(lin / sz / sy);
    // bricks begin at the first cell that may hold points: 1 in a padded table (the first brick, of the
    // padding alone, begins before the table)
    const int x0 = ((x + pad) & ~1) - pad, y0 = ((y + pad) & ~1) - pad, z0 = ((z + 3 * pad) & ~3) - 3 * pad;
    const uint32_t za = uint32_t(max(z0, 0)), zb = uint32_t(min(z0 + 4, span.z));
    uint32_t row = __ldg(&start[uint32_t(max(x0, 0)) * sy * sz]);
#pragma unroll
    for (int dx = 0; dx < 2; ++dx) {
        if (uint32_t(x0 + dx) >= uint32_t(span.x)) continue;
        const uint32_t slab = uint32_t(x0 + dx) * sy * sz;
        row += __ldg(&start[slab + uint32_t(max(y0, 0)) * sz]) - __ldg(&start[slab]);
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            if (uint32_t(y0 + dy) >= sy) continue;
            const uint32_t column = slab + uint32_t(y0 + dy) * sz;
            // columns before the cell's own in the quad count whole quads up to this one
            const uint32_t upto = 2 * dx + dy < 2 * (x - x0) + (y - y0) ? zb : za;
            row += __ldg(&start[column + upto]) - __ldg(&start[column]);
        }
    }
    return row + __ldg(&start[lin]) - __ldg(&start[lin - uint32_t(z) + za]);
}

// Final place = cell start + number of the cell's ids below this one's: the (cell, id) order
// of mod.rs:550, whatever order the atomics handed out the slots in.  order (optional): the walk
// order's row of each particle, its cell's row and its rank in the cell.
__global__ void k_rank_reorder(uint32_t n, const uint32_t* __restrict__ lin, const uint32_t* __restrict__ start,
                               const uint32_t* __restrict__ members, const uint32_t* __restrict__ ids_in,
                               const float4* __restrict__ pos_in, const float4* __restrict__ vel_in,
                               const float* __restrict__ rho_in, const int4* __restrict__ cells_in,
                               uint32_t* __restrict__ ids_out, float4* __restrict__ pos_out,
                               float4* __restrict__ vel_out, float* __restrict__ rho_out,
                               int4* __restrict__ cells_out, const float2* __restrict__ warm_in,
                               float2* __restrict__ warm_out, uint32_t skip_begin, uint32_t skip_end, Status* st,
                               uint32_t* __restrict__ dest, int3 span, int pad, uint32_t* __restrict__ order) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    // a job left undone (the fault injection of the dispatcher tests) places nothing; the count
    // of placed particles tells the host whether every particle was placed
    bool work = i < n && !(i >= skip_begin && i < skip_end);
    uint32_t placed = block_reduce(work ? 1u : 0u, SumU(), 0u);
    if (threadIdx.x == 0 && placed) atomicAdd(&st->processed, placed);
    if (i >= n) return;
    uint32_t l = lin[i];
    uint32_t b = start[l], e = start[l + 1];
    uint32_t id = ids_in[i];
    uint32_t rank = 0;
    for (uint32_t k = b; k < e; ++k) rank += members[k] < id ? 1u : 0u;
    uint32_t f = b + rank;
    if (order) order[walk_row(start, span, pad, l) + rank] = f;  // every row, a skipped job's too
    if (!work) return;
    if (dest) dest[i] = f;  // where each particle went, for the adjoint's way back
    ids_out[f] = id;
    pos_out[f] = pos_in[i];
    vel_out[f] = vel_in[i];
    rho_out[f] = rho_in[i];
    if (cells_in) cells_out[f] = cells_in[i];
    if (warm_in) warm_out[f] = warm_in[i];
}

// ---- exclusive scan of u32 in place, total written at data[m] ------------------------------

constexpr int kScanItems = 8;
constexpr int kScanTile = kBlock * kScanItems;
// tiles up to which each tile adds up its predecessors' sums itself (up to eight loads a thread)
constexpr uint32_t kScanOwnSums = 2048;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t warp_sums[kBlock / 32];
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < kBlock / 32 ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kBlock / 32) warp_sums[lane] = s;
    }
    __syncthreads();
    uint32_t warp_prefix = warp > 0 ? warp_sums[warp - 1] : 0u;
    if (total) *total = warp_sums[kBlock / 32 - 1];
    return warp_prefix + x - v;
}

// this thread's kScanItems of a tile at `base`; wide: the data is 16-byte aligned
__device__ __forceinline__ void scan_load(const uint32_t* data, uint32_t base, uint32_t m, bool wide,
                                          uint32_t (&v)[kScanItems]) {
    if (wide && base + kScanItems <= m) {
        const uint4 a = *reinterpret_cast<const uint4*>(data + base), b = *reinterpret_cast<const uint4*>(data + base + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        return;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] = base + k < m ? data[base + k] : 0u;
}
__device__ __forceinline__ void scan_store(uint32_t* data, uint32_t base, uint32_t m, bool wide,
                                           const uint32_t (&v)[kScanItems]) {
    if (wide && base + kScanItems <= m) {
        *reinterpret_cast<uint4*>(data + base) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(data + base + 4) = make_uint4(v[4], v[5], v[6], v[7]);
        return;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < m) data[base + k] = v[k];
}

__global__ void k_scan_tiles(uint32_t* data, uint32_t m, uint32_t* tile_sums, int wide) {
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems], out[kScanItems];
    scan_load(data, base, m, wide != 0, v);
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) sum += v[k];
    uint32_t total;
    uint32_t prefix = block_exclusive_scan(sum, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        out[k] = prefix;
        prefix += v[k];
    }
    scan_store(data, base, m, wide != 0, out);
    if (threadIdx.x == 0) {
        tile_sums[blockIdx.x] = total;
        if (gridDim.x == 1) data[m] = total;
    }
}

// Each tile adds up the sums of the tiles before it by itself (few enough of them that reading
// them again costs less than a launch that scans them) and adds that to its items: the scan 15.6
// -> 11 us at 1M (138 tiles), and 12 -> 6.5 where one tile holds the table.
__global__ void k_scan_finish(uint32_t* data, uint32_t m, const uint32_t* __restrict__ tile_sums, int wide) {
    __shared__ uint32_t before_s;
    uint32_t before = 0;
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kBlock) before += tile_sums[t];
    before = block_reduce(before, SumU(), 0u);
    if (threadIdx.x == 0) before_s = before;
    __syncthreads();
    before = before_s;
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    scan_load(data, base, m, wide != 0, v);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] += before;
    scan_store(data, base, m, wide != 0, v);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) data[m] = before + tile_sums[blockIdx.x];
}

// One block scans the tile sums (any count) in place.
__global__ void k_scan_sums(uint32_t* sums, uint32_t tiles) {
    __shared__ uint32_t carry_s;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (uint32_t base = 0; base < tiles; base += kBlock) {
        uint32_t i = base + threadIdx.x;
        uint32_t v = i < tiles ? sums[i] : 0u;
        uint32_t total;
        uint32_t x = block_exclusive_scan(v, &total);
        uint32_t carry = carry_s;
        if (i < tiles) sums[i] = x + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry_s = carry + total;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[tiles] = carry_s;  // grand total
}

__global__ void k_scan_add(uint32_t* data, uint32_t m, const uint32_t* __restrict__ tile_sums) {
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t add = tile_sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < m) data[base + k] += add;
    if (blockIdx.x == 0 && threadIdx.x == 0) data[m] = tile_sums[gridDim.x];
}

// ---- terrain (src/fluid/terrain.rs): the field's sampling is in fluid_device.cuh ---------------

// ground_near (mod.rs:657-663, terrain.rs:144-171, 305-310): the density the terrain regions
// holding the particle add, and the sum of their density gradients
__device__ __forceinline__ float ground_near(const TerrainDev& T, float px, float py, float pz, float3& slope) {
    float ground = 0.0f;
    slope = make_float3(0.0f, 0.0f, 0.0f);
    for (uint32_t r = 0; r < T.regions; ++r) {
        const TerrainRegion& t = T.region[r];
        float distance;
        float3 change;
        if (!terrain_read(T, t, px, py, pz, distance, change)) continue;
        float density = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f;
        if (distance < T.reach) {
            float open = distance - T.spacing / 2.0f;
            for (uint32_t k = 0; k < T.sites; ++k) {
                if (__ldg(&T.far[k]) <= open) continue;  // a distance moves no faster than the point
                float4 o = __ldg(&T.site[k]);
                float there;
                float3 toward;
                if (!terrain_read(T, t, px + o.x, py + o.y, pz + o.z, there, toward)) continue;
                float v = 0.5f - there / T.spacing;
                float share = v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);  // solid (terrain.rs:248-250)
                density += o.w * share;
                if (share > 0.0f && share < 1.0f) {
                    float w = o.w / T.spacing;
                    gx = gx - toward.x * w;
                    gy = gy - toward.y * w;
                    gz = gz - toward.z * w;
                }
            }
        }
        ground = ground + density;
        slope = make_float3(slope.x + gx, slope.y + gy, slope.z + gz);
    }
    return ground;
}

// ---- the density pass's two halves: the candidate scan, then the pair terms -------------------
// What bounds the pass: instruction issue and the latency of its gathers (the lists it writes are
// ~0.75 GB at 1M particles with kept gradients, 115 us at the copy rate).  Against a scan that
// branched per candidate, checked every cell's bounds, searched the walls' 27 cells for every
// particle, and divided three times a pair with one pair at a time (us, EXACT): 583 -> 433 (1M
// DFSPH), 198 -> 141 (250k DFSPH), 241 -> 159 (315k WCSPH), 474 -> 304 (64k WCSPH at support 4),
// 87 -> 59 (75k WCSPH).
// Four candidates and two pairs in flight, at 64 registers and four blocks a SM: two candidates
// measured 470 us at 1M, six 522, eight 556 (spills; 497 at 109 registers and two blocks), four
// pairs 482, and 48 registers for five blocks 571.  A grid of at most two blocks a SM runs wide
// instead (eight candidates and four pairs in flight, up to 128 registers): it has no other warps
// to hide behind.  74k particles: 57 -> 48 us, at support 4 378 -> 302; 111k, three blocks a SM,
// stay.

// a / radius, rounded as the IEEE division rounds it, without one: y = RN(1 / r), q = RN(a y), and
// RN(q + (a - q r) y) in two fmas, after Markstein ("Computation of elementary functions on the IBM RISC
// System/6000", 1990).  Three operations against the division's ten or so.  His theorem wants q within an
// ulp of a / r, and with significands a, r in [1, 2) this q may miss by (a + 1) / 2 ulps where a < r.  So:
//   - within an ulp the remainder is exact, and the sum errs by |remainder| |y - 1 / r|, near a midpoint
//     r 2^-50 at most (in units where ulp(q) = 2^-24), while a quotient is 2^-48 / r or more from it.
//   - further off the remainder may round, by 2^-47, and the sum errs by 2.8 2^-48 at most; but a / r is
//     (2 - a) 2^-25 or more short of the midpoint an ulp and a half from q.  With a = 2 - k 2^-23 that is
//     k 2^-48, enough from k = 3 on; k = 1 has no r above it, and k = 2 only r = 2 - 2^-23, where it is
//     3 2^-48 against an error of 2.5 2^-48.
// (test_radius_division.py goes through all a for some hundred radii.)  The remainder must not underflow:
// the settings' radius is checked on the host (odd_radius) and numerators under 2^-100 divide.  LOW:
// whether the numerator may be so small (a distance is 0 or at least 2^-75).
template <bool LOW>
__device__ __forceinline__ f32x2 div_radius2(const Params& p, f32x2 a) {
    const f32x2 y = splat2(p.inv_radius);
    const f32x2 q = mul2(a, y);
    f32x2 r = fma2(fma2(splat2(-p.radius), q, a), y, q);
    bool plain = p.odd_radius != 0u;
    if (LOW) {
        float a0, a1;
        unpack2(a, a0, a1);
        // 0 < |a| < 2^-100, by the bits (zero wraps round)
        const uint32_t edge = (127u - 100u) << 23;
        plain = plain || (__float_as_uint(a0) & 0x7fffffffu) - 1u < edge - 1u ||
                (__float_as_uint(a1) & 0x7fffffffu) - 1u < edge - 1u;
    }
    if (plain) {
        float a0, a1;
        unpack2(a, a0, a1);
        r = pack2(a0 / p.radius, a1 / p.radius);
    }
    return r;
}

// Kernel::value and the gradient factor (kernel_value, kernel_slope / d) of two pairs at squared
// distances d2, each half the scalar functions' bits.
__device__ __forceinline__ void kernel_pair(const Params& p, f32x2 d2, f32x2& value, float& g0, float& g1) {
    float s0, s1;
    unpack2(d2, s0, s1);
    // the particle itself (s = 0) stays off the slow paths of the root and the division
    const float r0 = sqrtf(s0 > 0.0f ? s0 : 1.0f), r1 = sqrtf(s1 > 0.0f ? s1 : 1.0f);
    const float d0 = s0 > 0.0f ? r0 : 0.0f, d1 = s1 > 0.0f ? r1 : 0.0f;
    const f32x2 q = div_radius2<false>(p, pack2(d0, d1));
    const f32x2 one = splat2(1.0f);
    const f32x2 om = fma2(q, splat2(-1.0f), one);  // 1 - q: the product is exact
    const f32x2 om2 = mul2(om, om);
    value = mul2(mul2(splat2(p.scale), mul2(om2, om2)), fma2(splat2(4.0f), q, one));  // 4 q is exact
    const f32x2 slope = div_radius2<true>(p, mul2(mul2(splat2(p.slope_scale), q), mul2(om, om2)));
    float l0, l1, q0, q1;
    unpack2(slope, l0, l1);
    unpack2(q, q0, q1);
    const bool p0 = q0 < 1.0f && d0 > 0.0f, p1 = q1 < 1.0f && d1 > 0.0f;
    g0 = (p0 ? l0 : 1.0f) / (p0 ? d0 : 1.0f);
    g1 = (p1 ? l1 : 1.0f) / (p1 ? d1 : 1.0f);
    g0 = p0 ? g0 : 0.0f;
    g1 = p1 ? g1 : 0.0f;
    if (!(q0 < 1.0f && q1 < 1.0f)) {  // at the very edge: value is zero from there on
        float v0, v1;
        unpack2(value, v0, v1);
        value = pack2(q0 < 1.0f ? v0 : 0.0f, q1 < 1.0f ? v1 : 0.0f);
    }
}

// The pair terms over a scanned list: for each of the first m indices in `from` (32 words apart),
// its entry {index, g} (and, with GRADIENT and room kept for it, its whole gradient G) goes to the
// row's list, and pair(v, gx, gy, gz) takes the kernel's value and G in list order.  Two pairs run
// packed, and the next ones' indices are requested before their terms are formed.  (`from` was
// written by this thread, and is rewritten for its next list: never a read-only load.)
template <bool GRADIENT, int U, class Pair>
__device__ __forceinline__ void pair_terms(const Params& p, const PairLists& l, uint32_t row, uint32_t m,
                                           const uint32_t* from, const float4* __restrict__ pts, float4 a,
                                           bool walls, Pair&& pair) {
    static_assert(U % 2 == 0, "pairs run two at a time");
    if (m == 0) return;
    uint2* e = l.e + l.at(row, 0);
    float4* gv = GRADIENT && l.gv ? l.gv + l.at(row, 0) : nullptr;
    uint32_t j[U];
#pragma unroll
    for (int u = 0; u < U; ++u) j[u] = from[size_t(u < (int)m ? u : m - 1) * 32u];
#pragma unroll 1
    for (uint32_t k = 0; k < m; k += U) {
        float4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) q[u] = __ldg(&pts[j[u]]);
        uint32_t next[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t kk = k + U + u;
            next[u] = from[size_t(kk < m ? kk : m - 1) * 32u];
        }
#pragma unroll
        for (int u = 0; u < U; u += 2) {
            const f32x2 ox = pack2(q[u].x - a.x, q[u + 1].x - a.x), oy = pack2(q[u].y - a.y, q[u + 1].y - a.y),
                        oz = pack2(q[u].z - a.z, q[u + 1].z - a.z);
            f32x2 value;
            float g[2], v[2];
            kernel_pair(p, sum2(p, sum2(p, mul2(ox, ox), mul2(oy, oy)), mul2(oz, oz)), value, g[0], g[1]);
            unpack2(value, v[0], v[1]);
            float gx[2] = {0.0f, 0.0f}, gy[2] = {0.0f, 0.0f}, gz[2] = {0.0f, 0.0f};
            if (GRADIENT) {
                // (at - other) g: both signs of the product turned, the same bits
                const f32x2 ng = pack2(-g[0], -g[1]);
                unpack2(mul2(ox, ng), gx[0], gx[1]);
                unpack2(mul2(oy, ng), gy[0], gy[1]);
                unpack2(mul2(oz, ng), gz[0], gz[1]);
            }
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                if (k + u + w < m) {
                    e[size_t(k + u + w) * 32u] = make_uint2(j[u + w], __float_as_uint(g[w]));
                    if (GRADIENT && gv)
                        gv[size_t(k + u + w) * 32u] =
                            make_float4(gx[w], gy[w], gz[w], walls ? 0.0f : __uint_as_float(j[u + w]));
                    pair(v[w], gx[w], gy[w], gz[w]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) j[u] = next[u];
    }
}

// ---- densities (mod.rs:621-675) and the substep's neighbour lists, with WCSPH pressure
// (step.rs:147-172) or the DFSPH factors (dfsph.rs:108-163) --------------------------------

// What the pass lists: the fluid (0), then the walls (1).
struct DensityIn {
    GridDev grid[2];
    const float4* pts[2];
    PairLists list[2];
};

// EXTRA: terrain regions or coupled bodies add their terms.  WIDE: two blocks a SM, else four (64 registers).
template <int SOLVER, bool EXTRA, bool WIDE>
__global__ void __launch_bounds__(kBlock, WIDE ? 2 : 4)
    k_density(const __grid_constant__ Params p, const __grid_constant__ DensityIn in, float* __restrict__ rho,
              float* __restrict__ press, float* __restrict__ scaled, float* __restrict__ alpha, Status* st, TerrainDev T,
              float4* __restrict__ slope, MoverDev M, uint32_t* scratch, PairRecords rec) {
    uint32_t compressed = 0, longest = 0;
    const float4* __restrict__ pos = in.pts[0];
    // this warp's unfinished list, entry k of a lane at k * 32: the same few megabytes for every row
    // the grid strides to, so the scan's stores stay in the L2 and only finished entries go to DRAM
    uint32_t* const idx = scratch + size_t(blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * 32u * in.list[0].cap +
                          (threadIdx.x & 31u);
    // rows of the walk order, a grid's width apart (one each when the grid covers them all)
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < p.n; row += gridDim.x * blockDim.x) {
        const uint32_t i = in.list[0].particle(row);
        float4 a = pos[i];
        int3 cell = cell_of(p, a.x, a.y, a.z);
        // The walk first only lists the neighbours (a tight loop over the ~216 candidates of 27
        // cells, of which ~16 % are kept), then takes the sums over the list, in list order, so
        // the arithmetic of the kept pairs runs without the candidates' divergence.  A list over
        // its room is incomplete and the host runs the pass again with more room.
        float sums[2], sx = 0.0f, sy = 0.0f, sz = 0.0f, squares = 0.0f;
#pragma unroll 1
        for (int w = 0; w < 2; ++w) {  // the fluid, then the walls
            const PairLists& l = in.list[w];
            const float4* __restrict__ pts = in.pts[w];
            const uint32_t found = scan_near<WIDE ? 8 : 4>(p, in.grid[w], pts, cell, a.x, a.y, a.z, idx, l.cap);
            l.count[row] = found;
            longest = max(longest, found);
            float sum = 0.0f;
            pair_terms<SOLVER == 1, WIDE ? 4 : 2>(p, l, row, found < l.cap ? found : l.cap, idx, pts, a, w == 1,
                                    [&](float v, float gx, float gy, float gz) {
                                        sum += v;
                                        if (SOLVER == 1) {  // factors (dfsph.rs:149-153); walls add no squares
                                            float px = gx * p.mass, py = gy * p.mass, pz = gz * p.mass;
                                            sx = sx + px;
                                            sy = sy + py;
                                            sz = sz + pz;
                                            squares += w == 0 ? dot3(px, py, pz, px, py, pz) : 0.0f;
                                        }
                                    });
            sums[1] = sum;
            if (w == 0) sums[0] = sum;
        }
        const float sum = sums[0], wsum = sums[1];
        // the coupled bodies' points, in their list order (mod.rs:648-656)
        float msum = 0.0f;
        if (EXTRA && M.count)
            each_near(p, M.grid, M.pos, cell, a.x, a.y, a.z, [&](uint32_t, float4 q) {
                float ox = q.x - a.x, oy = q.y - a.y, oz = q.z - a.z;
                msum += kernel_value(p, sqrtf(dot3(ox, oy, oz, ox, oy, oz)));
            });
        // mass (fluid + walls + body points) + ground (mod.rs:657-663)
        float3 gslope = make_float3(0.0f, 0.0f, 0.0f);
        float ground = EXTRA && T.regions ? ground_near(T, a.x, a.y, a.z, gslope) : 0.0f;
        float density = p.mass * (sum + wsum + msum) + ground;
        rho[i] = density;
        if (EXTRA && slope) slope[i] = make_float4(gslope.x, gslope.y, gslope.z, 0.0f);
        if (SOLVER == 0) {
            float ratio = fminf(density / p.rest, 1.1f);
            float pressure = fmaxf(p.stiffness * (pow7(ratio) - 1.0f), 0.0f);
            press[i] = pressure;
            const float over = pressure > p.divided_above ? pressure / (density * density) : 0.0f;
            scaled[i] = over;
            rec.pos_w[4 * size_t(i) + 3] = over;
        } else {
            float total = dot3(sx, sy, sz, sx, sy, sz) + squares;
            alpha[i] = total > 0.0f ? 1.0f / total : 0.0f;
        }
        rec.vel_w[4 * size_t(i) + 3] = density;
        float c = density / p.rest - 1.0f;
        if (c > 0.0f) compressed = max(compressed, __float_as_uint(c));
    }
    compressed = block_reduce(compressed, MaxU(), 0u);
    longest = block_reduce(longest, MaxU(), 0u);
    if (threadIdx.x == 0) {
        if (compressed) atomicMax(&st->maxcomp_bits, compressed);
        if (longest) atomicMax(&st->list_max, longest);
    }
}

// ---- scenes too small for a thread a row: L lanes a row -----------------------------------------
// A thread a row leaves a scene of 64,000 particles 13 warps a SM, each with one long chain of
// gathers, divisions and ordered adds; 8,000 particles leave most schedulers without a warp.  Here a warp takes 32 / L rows (lane = row + (32 / L) * sub,
// so that a step's list entries lie side by side), each lane every L-th candidate or pair; the terms
// meet in shared memory and one lane per (row, component) adds them in list order, so every sum is
// the one-thread walk's bit for bit.  A term past a list's end is +0, which leaves a sum that began
// at +0, and any value it is subtracted from, as it was.  Measured (density + force, us, against a
// warp a row whose lanes passed the terms round by shuffles): group_lanes.

constexpr int kGroupBlock = 128;
constexpr int kGroupBlocks = 8;  // a SM: 64 registers

template <int L, int NC>
struct GroupSums {
    static constexpr int kRows = 32 / L;
    static constexpr int kChunk = L < 16 ? 32 : 2 * L;  // pairs of a row between two rounds of adds
    static constexpr int kStride = kChunk + 4;          // 16-byte rows whose lanes fall in other banks
    static constexpr int kChains = kRows * NC;
    static constexpr int kRounds = (kChains + 31) / 32;
    float term[kChains * kStride];

    // this row's term c of its chunk's k-th pair
    __device__ __forceinline__ void put(int row, int c, int k, float v) { term[(row * NC + c) * kStride + k] = v; }

    // Adds (or, NEGATE, subtracts) the first `count` terms of every chain to its lane's acc, in order.
    template <bool NEGATE>
    __device__ __forceinline__ void add(float (&acc)[kRounds], uint32_t lane, uint32_t count) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
            if (lane + 32u * q < uint32_t(kChains)) {
                const float4* t = reinterpret_cast<const float4*>(term + (lane + 32u * q) * kStride);
                float s = acc[q];
#pragma unroll 4
                for (uint32_t k = 0; k < count; k += 4) {
                    const float4 v = t[k / 4];
                    s = NEGATE ? s - v.x : s + v.x;
                    s = NEGATE ? s - v.y : s + v.y;
                    s = NEGATE ? s - v.z : s + v.z;
                    s = NEGATE ? s - v.w : s + v.w;
                }
                acc[q] = s;
            }
        }
        __syncwarp();
    }

    // Every lane of a row gets the row's sums: out[c].
    __device__ __forceinline__ void spread(const float (&acc)[kRounds], uint32_t lane, int row, float (&out)[NC]) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kRounds; ++q)
            if (lane + 32u * q < uint32_t(kChains)) term[lane + 32u * q] = acc[q];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < NC; ++c) out[c] = term[row * NC + c];
        __syncwarp();
    }
};

// Appends the candidates that the L lanes of a row kept to its list: each lane had F of them one after
// another, its u-th the point j(u), kept where bit u of `kept` is set; the lists' order is the lanes'.
// nf, the list's length so far, is the same in every lane of the row.  (A ballot a candidate, the lanes
// interleaved, took 51 us for 8,000 particles at support 4 where this takes 48.5, and 195 against 189
// for 47k.  Where cells of few points are laid end to end the ballots stay: they were as fast.)
template <int L, int F, class J>
__device__ __forceinline__ void append_kept(uint32_t kept, J&& j, uint32_t* out, uint32_t cap, uint32_t lane, uint32_t& nf) {
    constexpr uint32_t R = 32u / L;
    if (!__any_sync(0xffffffffu, kept)) return;  // (most points of the outer cells)
    const uint32_t mine = uint32_t(__popc(kept));
    uint32_t upto = mine;
#pragma unroll
    for (int d = 1; d < L; d <<= 1) {
        const uint32_t other = __shfl_up_sync(0xffffffffu, upto, d * int(R));
        if (lane / R >= uint32_t(d)) upto += other;
    }
    uint32_t at = nf + upto - mine;
    nf += __shfl_sync(0xffffffffu, upto, 32u - R + lane % R);
#pragma unroll
    for (int u = 0; u < F; ++u) {
        if (kept >> u & 1u) {
            if (at < cap) out[size_t(at) * R] = j(u);
            ++at;
        }
    }
}

// scan_near by the L lanes of a row, for cells of many points: the list goes to out[k * 32 / L], the
// count comes back in every lane.  The warp walks the cells that any of its rows visits together, the
// lanes of a row testing L points of its cell at a time, kFlight of them each in flight.
template <int L, int kFlight>
__device__ __forceinline__ uint32_t scan_cells_group(const Params& p, const GridDev& g, const float4* __restrict__ pts,
                                                    bool valid, int3 cell, float x, float y, float z, uint32_t* out,
                                                    uint32_t cap, uint32_t lane) {
    constexpr uint32_t R = 32u / L;
    if (g.mode == 0) return 0u;
    const uint32_t sub = lane / R;
    const long long bx = (long long)cell.x - g.lx, by = (long long)cell.y - g.ly, bz = (long long)cell.z - g.lz;
    const int edge = g.near ? 0 : 1;
    const bool plain = g.mode == 1 && bx >= edge && bx + edge < g.sx && by >= edge && by + edge < g.sy && bz >= edge &&
                       bz + edge < g.sz;
    const f32x2 axy = pack2(-x, -y);
    const float az = -z;
    const uint32_t slab = uint32_t(g.sy) * uint32_t(g.sz);
    const uint32_t c0 = (uint32_t(bx) * uint32_t(g.sy) + uint32_t(by)) * uint32_t(g.sz) + uint32_t(bz);
    const uint32_t mine = !valid || !plain ? 0u : g.near ? __ldg(&g.near[c0]) : (1u << 27) - 1u;
    const ulonglong2* __restrict__ q2 = reinterpret_cast<const ulonglong2*>(pts);
    uint32_t nf = 0;
#pragma unroll 1
    for (uint32_t mask = __reduce_or_sync(0xffffffffu, mine); mask; mask &= mask - 1u) {
        const int t = __ffs(int(mask)) - 1;
        uint32_t b = 0, e = 0;
        if (mine >> t & 1u) {
            const uint32_t c = c0 + uint32_t((t % 3 - 1) * int(slab) + (t / 3 % 3 - 1) * g.sz + t / 9 - 1);
            b = __ldg(&g.start[c]);
            e = __ldg(&g.start[c + 1]);
        }
        const uint32_t longest = __reduce_max_sync(0xffffffffu, e - b);
#pragma unroll 1
        for (uint32_t k = 0; k < longest; k += uint32_t(kFlight * L)) {
            const uint32_t j0 = b + k + sub * uint32_t(kFlight);
            ulonglong2 q[kFlight];
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                if (j0 + u < e) q[u] = __ldg(q2 + j0 + u);
            }
            uint32_t kept = 0;
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                const f32x2 oxy = add2(f32x2{q[u].x}, axy);
                const float oz = __uint_as_float(uint32_t(q[u].y)) + az;
                float x2, y2;
                unpack2(mul2(oxy, oxy), x2, y2);
                if (j0 + u < e && (x2 + y2) + oz * oz < p.reach) kept |= 1u << u;
            }
            append_kept<L, kFlight>(kept, [&](int u) { return j0 + u; }, out, cap, lane, nf);
        }
    }
    if (__any_sync(0xffffffffu, valid && !plain)) {  // tables that need checks: one lane a row
        if (valid && !plain && sub == 0) nf = scan_checked(p, g, pts, cell, x, y, z, out, cap, R);
        nf = __shfl_sync(0xffffffffu, nf, lane % R);
    }
    return nf;
}

// The 27 cells around each row of a warp, laid end to end: cell c's points are candidates
// [upto[c - 1], upto[c]), point = candidate + shift[c].
template <int L>
struct GroupCells {
    static constexpr int kRows = 32 / L;
    uint32_t upto[kRows][28], shift[kRows][28];
};

// The same for cells of few points.  The lanes look the 27 cells up side by side, then test L candidates of the cells laid end
// to end at a time (kFlight of them each in flight) and place the kept ones by a ballot.
template <int L>
__device__ __forceinline__ uint32_t scan_near_group(const Params& p, const GridDev& g, const float4* __restrict__ pts,
                                                    bool valid, int3 cell, float x, float y, float z, uint32_t* out,
                                                    uint32_t cap, uint32_t lane, GroupCells<L>& cells) {
    constexpr uint32_t R = 32u / L;
    constexpr int kPer = (27 + L - 1) / L;  // cells a lane
    constexpr int kFlight = L <= 8 ? 4 : 2;
    if (g.mode == 0) return 0u;
    const uint32_t r = lane % R, sub = lane / R;
    const uint32_t own = (L == 32 ? 0xffffffffu : L == 16 ? 0x55555555u : L == 8 ? 0x11111111u : 0x01010101u) << r;
    const uint32_t below = own & ((1u << lane) - 1u);
    const long long bx = (long long)cell.x - g.lx, by = (long long)cell.y - g.ly, bz = (long long)cell.z - g.lz;
    const int edge = g.near ? 0 : 1;
    const bool plain = g.mode == 1 && bx >= edge && bx + edge < g.sx && by >= edge && by + edge < g.sy && bz >= edge &&
                       bz + edge < g.sz;
    const uint32_t slab = uint32_t(g.sy) * uint32_t(g.sz);
    const uint32_t c0 = (uint32_t(bx) * uint32_t(g.sy) + uint32_t(by)) * uint32_t(g.sz) + uint32_t(bz);
    const uint32_t mask = !valid || !plain ? 0u : g.near ? __ldg(&g.near[c0]) : (1u << 27) - 1u;
    uint32_t nf = 0;
    if (__any_sync(0xffffffffu, mask != 0u)) {
        uint32_t begin[kPer], len[kPer], total = 0;
#pragma unroll
        for (int c = 0; c < kPer; ++c) {
            const int t = int(sub) * kPer + c;
            begin[c] = len[c] = 0u;
            if (t < 27 && (mask >> t & 1u)) {
                const uint32_t at = c0 + uint32_t((t % 3 - 1) * int(slab) + (t / 3 % 3 - 1) * g.sz + t / 9 - 1);
                begin[c] = __ldg(&g.start[at]);
                len[c] = __ldg(&g.start[at + 1]) - begin[c];
            }
            total += len[c];
        }
        uint32_t upto = total;  // inclusive over the row's lanes
#pragma unroll
        for (int d = 1; d < L; d <<= 1) {
            const uint32_t other = __shfl_up_sync(0xffffffffu, upto, d * int(R));
            if (int(sub) >= d) upto += other;
        }
        const uint32_t all = __shfl_sync(0xffffffffu, upto, 32u - R + r);
        upto -= total;
#pragma unroll
        for (int c = 0; c < kPer; ++c) {
            const int t = int(sub) * kPer + c;
            if (t < 27) {
                cells.shift[r][t] = begin[c] - upto;
                upto += len[c];
                cells.upto[r][t] = upto;
            }
        }
        __syncwarp();
        const f32x2 axy = pack2(-x, -y);
        const float az = -z;
        const ulonglong2* __restrict__ q2 = reinterpret_cast<const ulonglong2*>(pts);
        const uint32_t most = __reduce_max_sync(0xffffffffu, all);
        uint32_t c = 0, end = cells.upto[r][0];
#pragma unroll 1
        for (uint32_t k = sub; k < most + sub; k += uint32_t(kFlight * L)) {  // (every lane the same rounds)
            ulonglong2 q[kFlight];
            uint32_t j[kFlight];
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                const uint32_t t = k + u * L;
                if (t < all) {
                    while (t >= end) end = cells.upto[r][++c];
                    j[u] = t + cells.shift[r][c];
                    q[u] = __ldg(q2 + j[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                const f32x2 oxy = add2(f32x2{q[u].x}, axy);
                const float oz = __uint_as_float(uint32_t(q[u].y)) + az;
                float x2, y2;
                unpack2(mul2(oxy, oxy), x2, y2);
                const bool keep = k + u * L < all && (x2 + y2) + oz * oz < p.reach;
                const uint32_t kept = __ballot_sync(0xffffffffu, keep);
                const uint32_t at = nf + __popc(kept & below);
                if (keep && at < cap) out[size_t(at) * R] = j[u];
                nf += __popc(kept & own);
            }
        }
        __syncwarp();
    }
    if (__any_sync(0xffffffffu, valid && !plain)) {  // tables that need checks: one lane a row
        if (valid && !plain && sub == 0) nf = scan_checked(p, g, pts, cell, x, y, z, out, cap, R);
        nf = __shfl_sync(0xffffffffu, nf, r);
    }
    return nf;
}

// k_density by L lanes a row.
// BODIES: coupled bodies add their points.  (Terrain keeps a thread a row.)
// FLIGHT: the scan a cell at a time with that many points a lane in flight (scan_cells_group); 0: the
// cells end to end (scan_near_group).
template <int SOLVER, bool BODIES, int L, int FLIGHT>
__global__ void __launch_bounds__(kGroupBlock, kGroupBlocks)
    k_density_group(const __grid_constant__ Params p, const __grid_constant__ DensityIn in, float* __restrict__ rho,
                    float* __restrict__ press, float* __restrict__ scaled, float* __restrict__ alpha, Status* st,
                    MoverDev M, uint32_t* scratch, PairRecords rec) {
    // the sums: the kernel's value, and with DFSPH the gradients' x, y, z and squares
    constexpr int NC = SOLVER == 1 ? 5 : 1, X = NC > 1 ? 1 : 0, Y = 2 * X, Z = 3 * X, Q = 4 * X;
    using Sums = GroupSums<L, NC>;
    constexpr uint32_t R = Sums::kRows;
    __shared__ __align__(16) Sums shared[kGroupBlock / 32];
    __shared__ GroupCells<L> cells[FLIGHT == 0 ? kGroupBlock / 32 : 1];
    Sums& S = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, r = lane % R, sub = lane / R;
    const uint32_t warp = blockIdx.x * (kGroupBlock / 32) + (threadIdx.x >> 5);
    const float4* __restrict__ pos = in.pts[0];
    uint32_t* const idx = scratch + size_t(warp) * R * in.list[0].cap + r;
    uint32_t compressed = 0, longest = 0;
    if (warp * R < p.n) {  // whole warps
        const uint32_t row = warp * R + r;
        const bool valid = row < p.n;
        const uint32_t i = valid ? in.list[0].particle(row) : 0u;
        const float4 a = pos[i];
        const int3 cell = cell_of(p, a.x, a.y, a.z);
        float acc[Sums::kRounds], sums[2] = {0.0f, 0.0f}, out[NC];
#pragma unroll
        for (int q = 0; q < Sums::kRounds; ++q) acc[q] = 0.0f;
#pragma unroll 1
        for (int w = 0; w < 2; ++w) {  // the fluid, then the walls
            const PairLists& l = in.list[w];
            const float4* __restrict__ pts = in.pts[w];
            uint32_t found;
            if constexpr (FLIGHT == 0)
                found = scan_near_group<L>(p, in.grid[w], pts, valid, cell, a.x, a.y, a.z, idx, l.cap, lane,
                                           cells[threadIdx.x >> 5]);
            else
                found = scan_cells_group<L, FLIGHT>(p, in.grid[w], pts, valid, cell, a.x, a.y, a.z, idx, l.cap, lane);
            if (valid && sub == 0) l.count[row] = found;
            longest = max(longest, found);
            const uint32_t m = valid ? min(found, l.cap) : 0u, most = __reduce_max_sync(0xffffffffu, m);
            __syncwarp();  // the indices the row's other lanes wrote
#pragma unroll 1
            for (uint32_t k0 = 0; k0 < most; k0 += Sums::kChunk) {
                // whole rounds of 2 L pairs, so every term that is added was put
                const uint32_t here = min(most - k0, uint32_t(Sums::kChunk));
#pragma unroll 1
                for (uint32_t round = 0; round < here; round += 2u * L) {
                    const uint32_t k = k0 + round + sub;
                    uint32_t j[2];
                    float4 q[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) j[u] = k + u * L < m ? idx[size_t(k + u * L) * R] : 0u;
#pragma unroll
                    for (int u = 0; u < 2; ++u) q[u] = k + u * L < m ? __ldg(&pts[j[u]]) : a;
                    const f32x2 ox = pack2(q[0].x - a.x, q[1].x - a.x), oy = pack2(q[0].y - a.y, q[1].y - a.y),
                                oz = pack2(q[0].z - a.z, q[1].z - a.z);
                    f32x2 value;
                    float g[2], v[2], gx[2] = {0.0f, 0.0f}, gy[2] = {0.0f, 0.0f}, gz[2] = {0.0f, 0.0f};
                    kernel_pair(p, sum2(p, sum2(p, mul2(ox, ox), mul2(oy, oy)), mul2(oz, oz)), value, g[0], g[1]);
                    unpack2(value, v[0], v[1]);
                    if (SOLVER == 1) {
                        const f32x2 ng = pack2(-g[0], -g[1]);  // (at - other) g, as pair_terms forms it
                        unpack2(mul2(ox, ng), gx[0], gx[1]);
                        unpack2(mul2(oy, ng), gy[0], gy[1]);
                        unpack2(mul2(oz, ng), gz[0], gz[1]);
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const uint32_t ku = k + u * L;
                        const bool there = ku < m;
                        if (there) l.e[l.at(row, ku)] = make_uint2(j[u], __float_as_uint(g[u]));
                        S.put(r, 0, ku - k0, there ? v[u] : 0.0f);
                        if (SOLVER == 1) {
                            if (there && l.gv)
                                l.gv[l.at(row, ku)] =
                                    make_float4(gx[u], gy[u], gz[u], w == 1 ? 0.0f : __uint_as_float(j[u]));
                            // factors (dfsph.rs:149-153); walls add no squares
                            const float px = there ? gx[u] * p.mass : 0.0f, py = there ? gy[u] * p.mass : 0.0f,
                                        pz = there ? gz[u] * p.mass : 0.0f;
                            S.put(r, X, ku - k0, px);
                            S.put(r, Y, ku - k0, py);
                            S.put(r, Z, ku - k0, pz);
                            S.put(r, Q, ku - k0, w == 0 ? dot3(px, py, pz, px, py, pz) : 0.0f);
                        }
                    }
                }
                S.template add<false>(acc, lane, here);
            }
            S.spread(acc, lane, int(r), out);
            sums[w] = out[0];
#pragma unroll
            for (int q = 0; q < Sums::kRounds; ++q)
                if ((lane + 32u * q) % uint32_t(NC) == 0u) acc[q] = 0.0f;  // the walls' values sum on their own
        }
        // the coupled bodies' points, in their list order (mod.rs:648-656)
        float msum = 0.0f;
        if (BODIES && valid && sub == 0)
            each_near(p, M.grid, M.pos, cell, a.x, a.y, a.z, [&](uint32_t, float4 q) {
                float ox = q.x - a.x, oy = q.y - a.y, oz = q.z - a.z;
                msum += kernel_value(p, sqrtf(dot3(ox, oy, oz, ox, oy, oz)));
            });
        if (valid && sub == 0) {
            float density = p.mass * (sums[0] + sums[1] + msum) + 0.0f;  // no ground
            rho[i] = density;
            if (SOLVER == 0) {
                float ratio = fminf(density / p.rest, 1.1f);
                float pressure = fmaxf(p.stiffness * (pow7(ratio) - 1.0f), 0.0f);
                press[i] = pressure;
                const float over = pressure > p.divided_above ? pressure / (density * density) : 0.0f;
                scaled[i] = over;
                rec.pos_w[4 * size_t(i) + 3] = over;
            } else {
                float total = dot3(out[X], out[Y], out[Z], out[X], out[Y], out[Z]) + out[Q];
                alpha[i] = total > 0.0f ? 1.0f / total : 0.0f;
            }
            rec.vel_w[4 * size_t(i) + 3] = density;
            float c = density / p.rest - 1.0f;
            if (c > 0.0f) compressed = max(compressed, __float_as_uint(c));
        }
    }
    compressed = block_reduce(compressed, MaxU(), 0u);
    longest = block_reduce(longest, MaxU(), 0u);
    if (threadIdx.x == 0) {
        if (compressed) atomicMax(&st->maxcomp_bits, compressed);
        if (longest) atomicMax(&st->list_max, longest);
    }
}

// Walks particle i's list: f(j, g, q) for each neighbour in list order, q = pts[j].  Entries are
// taken kListUnroll at a time, their gathers issued before any is used, and the next group's
// entries are requested before this group is used; past the end of the list the last entry is
// loaded again (a valid address) but not used, so the sums see exactly the list's terms in its
// order.
#ifndef SLF_LIST_UNROLL
#define SLF_LIST_UNROLL 4
#endif
constexpr int kListUnroll = SLF_LIST_UNROLL;
constexpr int kViscousBlock = 128;
// Resident blocks a SM that the solver's check and push are compiled for (caps their registers: check 64
// and 79, push 48 and 60).  Where the grid fills no more than three blocks a SM the registers are worth
// more than the warps, which there are none of: kFewBlocks, without spills and with more gathers in
// flight.  us, check and push, at the blocks for large grids / for few (and before the check lost its
// other walk, when it took 76 registers to gather ahead):
//     6,000 of support 4    58.6, 47.0 / 52.5, 45.0 (50.5, 45.4)     4,000  51.7, 39.3 / 44.7, 38.0 (46.5, 41.4)
//     15,000 of support 3   35.1, 25.9 / 30.9, 25.1 (33.4, 27.1)    60,000 45.7, 37.1 / 43.3, 35.6 (45.5, 35.4)
//     100,000 of support 2  22.9, 16.3 / 22.9, 14.9 (23.2, 16.9)    150,000 27.0, 18.9 / 31.2, 18.9
// and the push of 500k, 729k and 360k of support 3 41.3, 54.6, 90.2 / 43.5, 58.2, 101.
constexpr int kRateBlocks = 4, kPushBlocks = 5, kFewBlocks = 3;

template <class F>
__device__ __forceinline__ void each_listed(const PairLists& l, uint32_t i, const float4* __restrict__ pts, F&& f) {
    uint32_t n = l.count[i];
    if (n > l.cap) n = l.cap;
    if (n == 0) return;
    const uint2* __restrict__ base = l.e + l.at(i, 0);
    uint2 e[kListUnroll];
#pragma unroll
    for (int u = 0; u < kListUnroll; ++u) e[u] = SLF_LIST_LOAD(base + size_t(u < (int)n ? u : n - 1) * 32u);
    for (uint32_t k = 0; k < n; k += kListUnroll) {
        float4 q[kListUnroll];
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u) q[u] = __ldg(&pts[e[u].x]);
        uint2 next[kListUnroll];
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u) {
            uint32_t kk = k + kListUnroll + u;
            next[u] = SLF_LIST_LOAD(base + size_t(kk < n ? kk : n - 1) * 32u);
        }
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u)
            if (k + u < n) f(e[u].x, __uint_as_float(e[u].y), q[u]);
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u) e[u] = next[u];
    }
}

// The same walk with a second array gathered alongside (velocities).
template <class F>
__device__ __forceinline__ void each_listed2(const PairLists& l, uint32_t i, const float4* __restrict__ pts,
                                             const float4* __restrict__ more, F&& f) {
    uint32_t n = l.count[i];
    if (n > l.cap) n = l.cap;
    if (n == 0) return;
    const uint2* __restrict__ base = l.e + l.at(i, 0);
    uint2 e[kListUnroll];
#pragma unroll
    for (int u = 0; u < kListUnroll; ++u) e[u] = SLF_LIST_LOAD(base + size_t(u < (int)n ? u : n - 1) * 32u);
    for (uint32_t k = 0; k < n; k += kListUnroll) {
        float4 q[kListUnroll], w[kListUnroll];
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u) {
            q[u] = __ldg(&pts[e[u].x]);
            w[u] = __ldg(&more[e[u].x]);
        }
        uint2 next[kListUnroll];
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u) {
            uint32_t kk = k + kListUnroll + u;
            next[u] = SLF_LIST_LOAD(base + size_t(kk < n ? kk : n - 1) * 32u);
        }
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u)
            if (k + u < n) f(e[u].x, __uint_as_float(e[u].y), q[u], w[u]);
#pragma unroll
        for (int u = 0; u < kListUnroll; ++u) e[u] = next[u];
    }
}

// The solver check's walk, w = vel[index], the entries streamed evict-first and requested a group
// ahead.  Each slot takes one of two forms: slot k reads its kept gradient (PairLists::gv; 16 bytes, then one gather: the neighbour's velocity) when bit k % 4 of GV_SLOTS is set, and its
// {index, g} entry (8 bytes, then two gathers: position and velocity, G = (a - q) g as the
// density pass formed it) when not.  The first form moves more list bytes, the second gathers
// more: mixing them balances the pass's DRAM stream against its gathers.  f(G, w) in list order.
#ifndef SLF_RATE_GV_SLOTS
#define SLF_RATE_GV_SLOTS 0x7u
#endif
template <uint32_t GV_SLOTS, class F>
__device__ __forceinline__ void each_gradient_mixed(const PairLists& l, uint32_t row, const float4* __restrict__ pos,
                                                    const float4* __restrict__ vel, float4 a, F&& f) {
    static_assert(kListUnroll == 4, "slot forms repeat every four slots");
    uint32_t n = l.count[row];
    if (n > l.cap) n = l.cap;
    if (n == 0) return;
    const float4* __restrict__ gb = l.gv + l.at(row, 0);
    const uint2* __restrict__ eb = l.e + l.at(row, 0);
    float4 eg[4];
    uint2 ee[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        size_t kk = size_t(u < (int)n ? u : n - 1) * 32u;  // past the end: the last slot again, unused
        if (GV_SLOTS >> u & 1u) eg[u] = SLF_LIST_LOAD(gb + kk);
        else ee[u] = SLF_LIST_LOAD(eb + kk);
    }
    for (uint32_t k = 0; k < n; k += 4) {
        float4 q[4], w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (GV_SLOTS >> u & 1u) {
                w[u] = __ldg(&vel[__float_as_uint(eg[u].w)]);
            } else {
                q[u] = __ldg(&pos[ee[u].x]);
                w[u] = __ldg(&vel[ee[u].x]);
            }
        }
        float4 ng[4];
        uint2 ne[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            uint32_t kk = k + 4 + u;
            size_t at = size_t(kk < n ? kk : n - 1) * 32u;
            if (GV_SLOTS >> u & 1u) ng[u] = SLF_LIST_LOAD(gb + at);
            else ne[u] = SLF_LIST_LOAD(eb + at);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (k + u < n) {
                if (GV_SLOTS >> u & 1u) {
                    f(eg[u], w[u]);
                } else {
                    const float g = __uint_as_float(ee[u].y);
                    const float rx = a.x - q[u].x, ry = a.y - q[u].y, rz = a.z - q[u].z;
                    f(make_float4(rx * g, ry * g, rz * g, 0.0f), w[u]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (GV_SLOTS >> u & 1u) eg[u] = ng[u];
            else ee[u] = ne[u];
        }
    }
}

// The same over wall gradient entries, which need no gather (walls do not move): f(G).
template <class F>
__device__ __forceinline__ void each_wall_gradient(const PairLists& l, uint32_t row, F&& f) {
    uint32_t n = l.count[row];
    if (n > l.cap) n = l.cap;
    const float4* __restrict__ base = l.gv + l.at(row, 0);
#pragma unroll 4
    for (uint32_t k = 0; k < n; ++k) f(SLF_LIST_LOAD(base + size_t(k) * 32u));
}

// ---- wall viscosity (step.rs:262-301) -----------------------------------------------------

__device__ __forceinline__ float3 wall_viscous(const Params& p, float wall_visc, const PairLists& wl,
                                               const float4* __restrict__ walls, uint32_t row, float4 a, float4 v,
                                               float density, const TerrainDev& T) {
    if (wl.count[row] == 0 && T.regions == 0) return make_float3(0.0f, 0.0f, 0.0f);
    float awx = 0.0f, awy = 0.0f, awz = 0.0f;
    each_listed(wl, row, walls, [&](uint32_t, float g, float4 q) {
        float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
        awx = awx + -(rx * g);
        awy = awy + -(ry * g);
        awz = awz + -(rz * g);
    });
    // normalize_or(ZERO) dividing by the length
    float len = sqrtf(dot3(awx, awy, awz, awx, awy, awz));
    float nx = 0.0f, ny = 0.0f, nz = 0.0f;
    if (isfinite(len) && len > 0.0f) {
        nx = awx / len;
        ny = awy / len;
        nz = awz / len;
    }
    float k = fminf(dot3(v.x, v.y, v.z, nx, ny, nz), 0.0f);
    float ix = nx * k, iy = ny * k, iz = nz * k;
    float px = 0.0f, py = 0.0f, pz = 0.0f;
    // the ground damps the velocity into it by the weight of frozen water at that distance
    for (uint32_t r = 0; r < T.regions; ++r) {
        float distance;
        float3 gn;
        if (!terrain_sample(T, T.region[r], a.x, a.y, a.z, distance, gn)) continue;
        float into = dot3(v.x, v.y, v.z, gn.x, gn.y, gn.z);
        if (into < 0.0f) {
            float weight = ground_damping(T, distance);
            float c = wall_visc * into * weight / density;
            px = px - gn.x * c;
            py = py - gn.y * c;
            pz = pz - gn.z * c;
        }
    }
    each_listed(wl, row, walls, [&](uint32_t, float g, float4 q) {
        float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
        float toward = dot3(ix, iy, iz, rx, ry, rz);
        if (toward < 0.0f) {
            float squeeze = toward / (dot3(rx, ry, rz, rx, ry, rz) + p.soften);
            float damp = -wall_visc * squeeze / density;
            float s = p.mass * damp;
            px = px - (rx * g) * s;
            py = py - (ry * g) * s;
            pz = pz - (rz * g) * s;
        }
    });
    return make_float3(px, py, pz);
}

// ---- advance (step.rs:305-339) --------------------------------------------------------------

// terrain_contact (terrain.rs:314-333): each region in turn; true when the particle got under a
// surface.
__device__ __forceinline__ bool terrain_contact(const TerrainDev& T, float rest, float& nx, float& ny, float& nz,
                                                float4& v) {
    bool under = false;
    for (uint32_t r = 0; r < T.regions; ++r) contact_region(T, T.region[r], rest, nx, ny, nz, v, under);
    return under;
}

// zeroed (optional): the components the container's clamp held (bits x, y, z), whose position
// and velocity it set; terrain contact, after it, is not counted
__device__ __forceinline__ void advance_one(const Params& p, float dt, float4& a, float4& v, uint32_t& held,
                                            uint32_t& bad, const TerrainDev& T, uint32_t* zeroed = nullptr) {
    float nx = a.x + v.x * dt, ny = a.y + v.y * dt, nz = a.z + v.z * dt;
    if (p.has_bounds) {
        float ix = fminf(fmaxf(nx, p.low_in.x), p.high_in.x);
        float iy = fminf(fmaxf(ny, p.low_in.y), p.high_in.y);
        float iz = fminf(fmaxf(nz, p.low_in.z), p.high_in.z);
        if (ix != nx || iy != ny || iz != nz) {
            float cx = fminf(fmaxf(nx, p.low.x), p.high.x);
            float cy = fminf(fmaxf(ny, p.low.y), p.high.y);
            float cz = fminf(fmaxf(nz, p.low.z), p.high.z);
            if (cx != nx || cy != ny || cz != nz) held += 1;
            if (zeroed) *zeroed = (ix != nx ? 1u : 0u) | (iy != ny ? 2u : 0u) | (iz != nz ? 4u : 0u);
            if (ix != nx) v.x = 0.0f;
            if (iy != ny) v.y = 0.0f;
            if (iz != nz) v.z = 0.0f;
            nx = ix;
            ny = iy;
            nz = iz;
        }
    }
    if (T.regions && terrain_contact(T, p.spacing / 2.0f, nx, ny, nz, v)) held += 1;
    if (!(isfinite(nx) && isfinite(ny) && isfinite(nz) && isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) bad = 1;
    a.x = nx;
    a.y = ny;
    a.z = nz;
}

// ---- coupled bodies' points (couple.rs:375-416) ---------------------------------------------

// The body points within reach of a particle at `a` moving at `v`, in list order: for each,
// f(j, gradient * mass (xyz), mirrored + damp, damp, toward) with the reference's arithmetic.
template <class F>
__device__ __forceinline__ void mover_pairs(const Params& p, const MoverDev& M, float damping, float4 a, float4 v,
                                            float density, float mirrored, F&& f) {
    int3 cell = cell_of(p, a.x, a.y, a.z);
    each_near(p, M.grid, M.pos, cell, a.x, a.y, a.z, [&](uint32_t j, float4 q) {
        float ox = a.x - q.x, oy = a.y - q.y, oz = a.z - q.z;  // at - point
        float4 w = __ldg(&M.vel[j]);
        float toward = dot3(v.x - w.x, v.y - w.y, v.z - w.z, ox, oy, oz);
        float damp = toward < 0.0f ? -damping * toward / (dot3(ox, oy, oz, ox, oy, oz) + p.soften) / density : 0.0f;
        float g = kernel_gradient_factor(p, ox, oy, oz);
        f(j, (ox * g) * p.mass, (oy * g) * p.mass, (oz * g) * p.mass, mirrored + damp, damp, toward);
    });
}

// What the body points took from the water this substep (couple.rs:401-414): per 512-particle chunk
// and body, the damping force and its torque about the body's centre, summed over the chunk's pairs in
// particle then pair order (step.rs:173-221).  Pairs below the settling speed give nothing.  A block a
// chunk: its threads count their particles' pairs, a scan places them, and the pairs go through shared
// memory kFeltPairs at a time, where one thread per (body, component) adds them in order.  Most chunks
// touch no body and end after the count.  felt[c * bodies + b] = (force, torque).
// (As counts, a scan, a host wait for their total, pair records in memory and a thread per chunk and
// body over them, before: five launches and a wait a substep.)
constexpr int kFeltBlock = 512, kFeltPairs = 256;

__global__ void __launch_bounds__(kFeltBlock) k_mover_felt(const __grid_constant__ Params p,
                                                           float mover_damping,
                                                           const __grid_constant__ MoverDev M,
                                                           const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                           const float* __restrict__ rho, const float* __restrict__ press,
                                                           const float* __restrict__ scaled,
                                                           const float4* __restrict__ centre, float elapsed,
                                                           uint32_t bodies, float4* __restrict__ felt) {
    __shared__ float term[6][kFeltPairs];
    __shared__ uint32_t owner[kFeltPairs];
    __shared__ uint32_t warp_sums[kFeltBlock / 32];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    float* const sums = reinterpret_cast<float*>(felt + 2 * size_t(blockIdx.x) * bodies);  // [b][8], 3 and 7 unused
    for (uint32_t q = t; q < 8u * bodies; q += kFeltBlock) sums[q] = 0.0f;
    const uint32_t i = blockIdx.x * uint32_t(kFeltBlock) + t;
    const bool valid = i < p.n;
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v = a;
    float density = 1.0f, mirrored = 0.0f;
    if (valid) {
        a = pos[i];
        v = vel[i];
        density = rho[i];
        mirrored = scaled[i] + (press[i] > p.divided_above ? press[i] / p.rest_sq : 0.0f);
    }
    // f(k, j, point, gradient * mass, damp) for the particle's k-th pair above the settling speed
    auto pairs = [&](auto&& f) {
        uint32_t k = 0;
        mover_pairs(p, M, mover_damping, a, v, density, mirrored,
                    [&](uint32_t j, float gx, float gy, float gz, float, float damp, float toward) {
                        const float4 q = __ldg(&M.pos[j]);
                        const float ox = a.x - q.x, oy = a.y - q.y, oz = a.z - q.z;
                        if (toward * toward < p.settles * dot3(ox, oy, oz, ox, oy, oz)) return;
                        f(k, q, gx, gy, gz, damp);
                        ++k;
                    });
        return k;
    };
    const uint32_t mine = valid ? pairs([](uint32_t, float4, float, float, float, float) {}) : 0u;
    // where the particle's pairs stand among the chunk's
    uint32_t upto = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t other = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= uint32_t(d)) upto += other;
    }
    __syncthreads();
    if (lane == 31) warp_sums[warp] = upto;
    __syncthreads();
    uint32_t before = upto - mine, total = 0;
#pragma unroll
    for (int w = 0; w < kFeltBlock / 32; ++w) {
        if (uint32_t(w) < warp) before += warp_sums[w];
        total += warp_sums[w];
    }
    for (uint32_t base = 0; base < total; base += kFeltPairs) {
        const uint32_t here = min(total - base, uint32_t(kFeltPairs));
        if (mine && before < base + here && before + mine > base)
            pairs([&](uint32_t k, float4 q, float gx, float gy, float gz, float damp) {
                const uint32_t at = before + k - base;  // (wraps past `here` before the window)
                if (at >= here) return;
                const uint32_t b = __float_as_uint(q.w);
                const float4 c = centre[2 * size_t(b)], u = centre[2 * size_t(b) + 1];
                const float cx = c.x + u.x * elapsed, cy = c.y + u.y * elapsed, cz = c.z + u.z * elapsed;
                const float s = damp * p.mass;
                const float ex = gx * s, ey = gy * s, ez = gz * s;
                const float rx = q.x - cx, ry = q.y - cy, rz = q.z - cz;
                term[0][at] = ex;
                term[1][at] = ey;
                term[2][at] = ez;
                term[3][at] = ry * ez - ey * rz;
                term[4][at] = rz * ex - ez * rx;
                term[5][at] = rx * ey - ex * ry;
                owner[at] = b;
            });
        __syncthreads();
        for (uint32_t q = t; q < 6u * bodies; q += kFeltBlock) {
            const uint32_t b = q / 6u, c = q % 6u;
            float* const to = sums + 8 * size_t(b) + c + (c >= 3u ? 1u : 0u);
            float sum = *to;
#pragma unroll 4
            for (uint32_t k = 0; k < here; ++k)
                if (owner[k] == b) sum = sum + term[c][k];
            *to = sum;
        }
        __syncthreads();
    }
}

// Whether any cell of the box [lo, hi] (cell keys) holds fluid in the last sort's dense table
// (couple.rs:350-357); *wet = 1 if so.
__global__ void k_cells_wet(GridDev g, int3 lo, int3 hi, uint32_t* wet) {
    long long nx = (long long)hi.x - lo.x + 1, ny = (long long)hi.y - lo.y + 1, nz = (long long)hi.z - lo.z + 1;
    long long total = nx * ny * nz;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        long long x = lo.x + t / (ny * nz), y = lo.y + (t / nz) % ny, z = lo.z + t % nz;
        uint32_t b, e;
        if (g.range(x, y, z, b, e)) {
            *wet = 1u;
            return;
        }
    }
}

// ---- WCSPH: forces, velocity update and advance in one pass (step.rs:159-223, 305-339) -----

// k_wcsph_force by L lanes a row.
template <bool BODIES, int L>
__global__ void __launch_bounds__(kGroupBlock, BODIES ? 9 : kGroupBlocks)
    k_wcsph_force_group(Params p, const StepConsts* __restrict__ sc, PairLists fl, PairLists wl,
                        const float4* __restrict__ pos, const float4* __restrict__ vel, const float* __restrict__ rho,
                        const float* __restrict__ press, const float* __restrict__ scaled,
                        const float4* __restrict__ walls, float4* __restrict__ pos_out, float4* __restrict__ vel_out,
                        Status* st, float4* __restrict__ vel_pre, MoverDev M) {
    using Sums = GroupSums<L, 3>;
    constexpr uint32_t R = Sums::kRows;
    __shared__ __align__(16) Sums shared[kGroupBlock / 32];
    Sums& S = shared[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, r = lane % R, sub = lane / R;
    const uint32_t warp = blockIdx.x * (kGroupBlock / 32) + (threadIdx.x >> 5);
    int3 lo = make_int3(INT_MAX, INT_MAX, INT_MAX), hi = make_int3(INT_MIN, INT_MIN, INT_MIN);
    float fastest = 0.0f;
    uint32_t held = 0, bad = 0;
    const float dt = sc->dt, visc = sc->viscosity, wall_visc = sc->wall_viscosity;
    if (warp * R < p.n) {  // whole warps
        const uint32_t row = warp * R + r;
        const bool valid = row < p.n;
        const uint32_t i = valid ? fl.particle(row) : 0u;
        float4 a = pos[i];
        float4 v = vel[i];
        const float density = rho[i], own = scaled[i];
        // every row's terms, in list order: term(k, entry, tx, ty, tz) for the row's k-th entry, and
        // the chains take what these pairs put
        auto walk = [&](const PairLists& l, auto negate, float(&acc)[Sums::kRounds], auto&& term) {
            const uint32_t m = valid ? min(l.count[row], l.cap) : 0u, most = __reduce_max_sync(0xffffffffu, m);
#pragma unroll 1
            for (uint32_t k0 = 0; k0 < most; k0 += Sums::kChunk) {
                const uint32_t here = min(most - k0, uint32_t(Sums::kChunk));
#pragma unroll 1
                for (uint32_t round = 0; round < here; round += 2u * L) {
                    const uint32_t k = k0 + round + sub;
                    uint2 en[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        en[u] = k + u * L < m ? SLF_LIST_LOAD(l.e + l.at(row, k + u * L)) : make_uint2(0u, 0u);
                    float t[2][3];
                    term(en, t);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const bool there = k + u * L < m;
#pragma unroll
                        for (int c = 0; c < 3; ++c) S.put(r, c, round + sub + u * L, there ? t[u][c] : 0.0f);
                    }
                }
                S.template add<decltype(negate)::value>(acc, lane, here);
            }
            return most;
        };
        float push[Sums::kRounds] = {}, away[Sums::kRounds] = {}, damped[Sums::kRounds] = {};
        walk(fl, std::true_type{}, push, [&](const uint2(&en)[2], float(&t)[2][3]) {
            float4 q[2], w[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) q[u] = __ldg(&pos[en[u].x]), w[u] = __ldg(&vel[en[u].x]);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float g = __uint_as_float(en[u].y);
                float rx = a.x - q[u].x, ry = a.y - q[u].y, rz = a.z - q[u].z;
                float squared = dot3(rx, ry, rz, rx, ry, rz);
                float gx = rx * g, gy = ry * g, gz = rz * g;
                float toward = dot3(v.x - w[u].x, v.y - w[u].y, v.z - w[u].z, rx, ry, rz);
                float damp = p.parted;  // a pair that parts: no division of a zero
                if (toward < 0.0f) damp = -visc * toward / (squared + p.soften) * 2.0f / (density + w[u].w);
                float s = p.mass * (own + q[u].w + damp);
                const bool pair = squared > 0.0f;
                t[u][0] = pair ? gx * s : 0.0f, t[u][1] = pair ? gy * s : 0.0f, t[u][2] = pair ? gz * s : 0.0f;
            }
        });
        const float mirrored = own + (press[i] > p.divided_above ? press[i] / p.rest_sq : 0.0f);
        // the walls' pressure, then wall_viscous's two walks (its normal, then its damping)
        const uint32_t walled = walk(wl, std::true_type{}, push, [&](const uint2(&en)[2], float(&t)[2][3]) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float g = __uint_as_float(en[u].y);
                const float4 q = __ldg(&walls[en[u].x]);
                float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
                float s = p.mass * mirrored;
                t[u][0] = (rx * g) * s, t[u][1] = (ry * g) * s, t[u][2] = (rz * g) * s;
            }
        });
        float sum[3], wall[3] = {0.0f, 0.0f, 0.0f};
        S.spread(push, lane, int(r), sum);
        if (walled) {
            walk(wl, std::false_type{}, away, [&](const uint2(&en)[2], float(&t)[2][3]) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float g = __uint_as_float(en[u].y);
                    const float4 q = __ldg(&walls[en[u].x]);
                    float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
                    t[u][0] = -(rx * g), t[u][1] = -(ry * g), t[u][2] = -(rz * g);
                }
            });
            float aw[3];
            S.spread(away, lane, int(r), aw);
            // wall_viscous (step.rs:262-301): normalize_or(ZERO) dividing by the length
            float len = sqrtf(dot3(aw[0], aw[1], aw[2], aw[0], aw[1], aw[2]));
            float ux = 0.0f, uy = 0.0f, uz = 0.0f;
            if (isfinite(len) && len > 0.0f) {
                ux = aw[0] / len;
                uy = aw[1] / len;
                uz = aw[2] / len;
            }
            float kk = fminf(dot3(v.x, v.y, v.z, ux, uy, uz), 0.0f);
            float ix = ux * kk, iy = uy * kk, iz = uz * kk;
            walk(wl, std::true_type{}, damped, [&](const uint2(&en)[2], float(&t)[2][3]) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float g = __uint_as_float(en[u].y);
                    const float4 q = __ldg(&walls[en[u].x]);
                    float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
                    float toward = dot3(ix, iy, iz, rx, ry, rz);
                    t[u][0] = t[u][1] = t[u][2] = 0.0f;
                    if (toward < 0.0f) {
                        float squeeze = toward / (dot3(rx, ry, rz, rx, ry, rz) + p.soften);
                        float damp = -wall_visc * squeeze / density;
                        float s = p.mass * damp;
                        t[u][0] = (rx * g) * s, t[u][1] = (ry * g) * s, t[u][2] = (rz * g) * s;
                    }
                }
            });
            S.spread(damped, lane, int(r), wall);
        }
        if (valid && sub == 0) {
            float px = sum[0], py = sum[1], pz = sum[2];
            if (BODIES)
                mover_pairs(p, M, sc->mover_damping, a, v, density, mirrored,
                            [&](uint32_t, float gx, float gy, float gz, float s, float, float) {
                                px = px - gx * s;
                                py = py - gy * s;
                                pz = pz - gz * s;
                            });
            float ax = (px + wall[0]) + p.gravity.x, ay = (py + wall[1]) + p.gravity.y, az = (pz + wall[2]) + p.gravity.z;
            v.x = v.x + ax * dt;
            v.y = v.y + ay * dt;
            v.z = v.z + az * dt;
            float4 pre = v;
            uint32_t flags = 0;
            advance_one(p, dt, a, v, held, bad, TerrainDev{}, &flags);
            if (vel_pre) {
                // the velocity before the wall zeroed any component, and which ones it zeroed
                pre.w = __uint_as_float(flags);
                vel_pre[i] = pre;
            }
            pos_out[i] = a;
            vel_out[i] = v;
            const int3 nc = cell_of(p, a.x, a.y, a.z);
            lo = make_int3(min(lo.x, nc.x), min(lo.y, nc.y), min(lo.z, nc.z));
            hi = make_int3(max(hi.x, nc.x), max(hi.y, nc.y), max(hi.z, nc.z));
            fastest = fmaxf(fastest, sqrtf(dot3(v.x, v.y, v.z, v.x, v.y, v.z)));
        }
    }
    fold_advance_box(st, lo, hi, fastest, held, bad);
}

// A thread a row, rows of the walk order a grid's width apart.  One 16-byte gather brings a
// neighbour's position and p / rho^2, another its velocity and density (four gathers before), and a
// pair that moves apart divides nothing: 157 -> 68 us at 262k particles (measured 157 -> 96 at 314k
// by the gathers and three blocks of 80 registers a SM; four blocks spill, 108; two 124), then
// 86 -> 68 at 262k and 249 -> 155 at 47k, support 4, by the division of zero (its slow path ran for
// half of all pairs).  EXTRA: terrain regions or
// coupled bodies add their terms.
template <bool EXTRA>
__global__ void __launch_bounds__(kBlock, 3) k_wcsph_force(Params p, const StepConsts* __restrict__ sc, PairLists fl,
                                                        PairLists wl, const float4* __restrict__ pos,
                                                        const float4* __restrict__ vel, const float* __restrict__ rho,
                                                        const float* __restrict__ press,
                                                        const float* __restrict__ scaled,
                                                        const float4* __restrict__ walls, float4* __restrict__ pos_out,
                                                        float4* __restrict__ vel_out, Status* st,
                                                        float4* __restrict__ vel_pre, TerrainDev T,
                                                        const float4* __restrict__ slope, MoverDev M) {
    int3 lo = make_int3(INT_MAX, INT_MAX, INT_MAX), hi = make_int3(INT_MIN, INT_MIN, INT_MIN);
    float fastest = 0.0f;
    uint32_t held = 0, bad = 0;
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < p.n; row += gridDim.x * blockDim.x) {
        const uint32_t i = fl.particle(row);
        const float dt = sc->dt;
        const float visc = sc->viscosity;
        float4 a = pos[i];
        float4 v = vel[i];
        float density = rho[i];
        float own = scaled[i];
        float px = 0.0f, py = 0.0f, pz = 0.0f;
        each_listed2(fl, row, pos, vel, [&](uint32_t, float g, float4 q, float4 w) {
            float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
            float squared = dot3(rx, ry, rz, rx, ry, rz);
            if (squared <= 0.0f) return;
            // g = slope(distance) / distance with distance = sqrt(squared) > 0; q.w is the
            // neighbour's p / rho^2 and w.w its density (the density pass put them there)
            float gx = rx * g, gy = ry * g, gz = rz * g;
            float toward = dot3(v.x - w.x, v.y - w.y, v.z - w.z, rx, ry, rz);
            float damp = p.parted;  // a pair that parts: no division of a zero
            if (toward < 0.0f) damp = -visc * toward / (squared + p.soften) * 2.0f / (density + w.w);
            float s = p.mass * (own + q.w + damp);
            px = px - gx * s;
            py = py - gy * s;
            pz = pz - gz * s;
        });
        float mirrored = own + (press[i] > p.divided_above ? press[i] / p.rest_sq : 0.0f);
        each_listed(wl, row, walls, [&](uint32_t, float g, float4 q) {
            float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
            float s = p.mass * mirrored;
            px = px - (rx * g) * s;
            py = py - (ry * g) * s;
            pz = pz - (rz * g) * s;
        });
        if (EXTRA && slope) {  // the ground pushes back with this particle's own pressure (step.rs:203-205)
            float4 sl = slope[i];
            px = px - sl.x * mirrored;
            py = py - sl.y * mirrored;
            pz = pz - sl.z * mirrored;
        }
        if (EXTRA && M.count)
            mover_pairs(p, M, sc->mover_damping, a, v, density, mirrored,
                        [&](uint32_t, float gx, float gy, float gz, float s, float, float) {
                            px = px - gx * s;
                            py = py - gy * s;
                            pz = pz - gz * s;
                        });
        TerrainDev none{};
        float3 wv = wall_viscous(p, sc->wall_viscosity, wl, walls, row, a, v, density, EXTRA ? T : none);
        float ax = (px + wv.x) + p.gravity.x, ay = (py + wv.y) + p.gravity.y, az = (pz + wv.z) + p.gravity.z;
        v.x = v.x + ax * dt;
        v.y = v.y + ay * dt;
        v.z = v.z + az * dt;
        float4 pre = v;
        uint32_t flags = 0;
        advance_one(p, dt, a, v, held, bad, EXTRA ? T : none, &flags);
        if (vel_pre) {
            // the velocity before the wall zeroed any component, and which ones it zeroed
            pre.w = __uint_as_float(flags);
            vel_pre[i] = pre;
        }
        pos_out[i] = a;
        vel_out[i] = v;
        const int3 nc = cell_of(p, a.x, a.y, a.z);
        lo = make_int3(min(lo.x, nc.x), min(lo.y, nc.y), min(lo.z, nc.z));
        hi = make_int3(max(hi.x, nc.x), max(hi.y, nc.y), max(hi.z, nc.z));
        const float speed = sqrtf(dot3(v.x, v.y, v.z, v.x, v.y, v.z));
        fastest = fmaxf(fastest, speed);  // (a NaN speed is ignored, as f32::max does)
    }
    fold_advance_box(st, lo, hi, fastest, held, bad);
}

// ---- DFSPH ----------------------------------------------------------------------------------

// density_rate (dfsph.rs:166-181), then the solve's stiffness and error (dfsph.rs:241-259) of
// particle i.  The lists always carry the kept gradients here, the walls' too: with no walk over
// {index, g} entries beside this one the pass keeps its registers (76 -> 4 bytes spilled at 64
// registers) and takes 106.2 us a launch at 1M, 37.9 at 250k, from 108.6 and 39.4.  Three blocks
// a SM take 107.3 and 41.4, five (100 bytes spilled) 129.7 and 48.9.
template <int WHICH>
__device__ __forceinline__ void rate_particle(const Params& p, const StepConsts* __restrict__ sc,
                                              const PairLists& fl, const PairLists& wl, uint32_t i, uint32_t row,
                                              const float4* __restrict__ pos, const float4* __restrict__ vel,
                                              const float* __restrict__ rho, const float* __restrict__ alpha,
                                              float* __restrict__ kappa_w,
                                              SolveRec rec, uint32_t slot, double& err, uint32_t& loaded) {
    const float dt = sc->dt;
    float4 a = pos[i];
    float4 v = vel[i];
    float rate = 0.0f;
    // the gradients the density pass kept, for the slots that read them
    each_gradient_mixed<SLF_RATE_GV_SLOTS>(fl, row, pos, vel, a, [&](float4 G, float4 w) {
        rate += dot3(v.x - w.x, v.y - w.y, v.z - w.z, G.x, G.y, G.z);
    });
    each_wall_gradient(wl, row, [&](float4 G) { rate += dot3(v.x, v.y, v.z, G.x, G.y, G.z); });
    rate = rate * p.mass;
    if (rec.rate) {  // recorded for the adjoint
        size_t at = size_t(slot) * p.n + i;
        rec.rate[at] = rate;
        rec.vel[at] = v;
    }
    float target, error;
    if (WHICH == 1) {
        float over = fmaxf(rho[i] + dt * rate - p.rest, 0.0f);
        // (a quotient of zero is zero, and its division would take the slow path)
        target = over > sc->divided_above ? over / sc->dt_sq : 0.0f;
        error = over > 0.0f ? over / p.rest : 0.0f;
    } else {
        float r = fl.count[row] + wl.count[row] < 20u ? 0.0f : fmaxf(rate, 0.0f);
        target = r > 0.0f ? r / dt : 0.0f;
        error = r > 0.0f ? dt * r / p.rest : 0.0f;
    }
    // the stiffness rides in the spare lane of the position, where push_apart gathers it
    kappa_w[4 * (size_t)i + 3] = target * alpha[i];
    err = (double)error;
    loaded = error > 0.0f ? 1u : 0u;
}

// One check of the solve, a particle a thread, and the average error of the particles under
// load (dfsph.rs:263-268) in a last-block finish.
template <int WHICH, int BLOCKS>
__global__ void __launch_bounds__(kBlock, BLOCKS) k_rate(Params p, const StepConsts* __restrict__ sc, PairLists fl,
                                                 PairLists wl, const float4* __restrict__ pos,
                                                 const float4* __restrict__ vel, const float* __restrict__ rho,
                                                 const float* __restrict__ alpha, float* __restrict__ kappa_w,
                                                 DD* __restrict__ partial,
                                                 uint32_t* __restrict__ partial_loaded, Status* st,
                                                 SolveRec rec, unsigned long long loop) {
    // a solve that already stopped leaves the rest of its batch of launches idle
    if (__ldcg(&st->settled)) return;
    DD acc{0.0, 0.0};
    uint32_t loaded = 0;
    // every block reads the count before the last block advances it
    const uint32_t slot = rec.rate ? __ldcg(&st->iterations) : 0u;
    // rows of the walk order, a grid's width apart (one each when the grid covers them all)
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < p.n; row += gridDim.x * blockDim.x) {
        const uint32_t i = fl.particle(row);
        double err = 0.0;
        uint32_t one = 0;
        rate_particle<WHICH>(p, sc, fl, wl, i, row, pos, vel, rho, alpha, kappa_w, rec, slot, err, one);
        acc = dd_add(acc, DD{err, 0.0});
        loaded += one;
    }
    residual_finish<WHICH>(p, st, partial, partial_loaded, acc, loaded, loop);
}

// push_apart (dfsph.rs:184-216) of particle i: the velocity change from each particle's
// stiffness, which the rate pass left in the w lane of each position.  Fluid pairs read {index, g}
// and gather that record: a kept gradient in the entry's place moves 8 bytes more for nothing,
// with the stiffness alone gathered too (1 to 4 slots in four: 78 to 100 us at 1M against 72).
// Wall pairs need no gather at all from their kept gradients: 72 -> 69 us.
__device__ __forceinline__ void push_particle(const Params& p, const StepConsts* __restrict__ sc, const PairLists& fl,
                                              const PairLists& wl, uint32_t i, uint32_t row,
                                              const float4* __restrict__ pos, float4* __restrict__ vel,
                                              float* __restrict__ applied) {
    const float dt = sc->dt;
    float4 a = pos[i];
    float own = a.w;
    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
    each_listed(fl, row, pos, [&](uint32_t, float g, float4 q) {
        float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
        float s = p.mass * (own + q.w);
        cx = cx - (rx * g) * s;
        cy = cy - (ry * g) * s;
        cz = cz - (rz * g) * s;
    });
    const float ws = p.mass * own;
    each_wall_gradient(wl, row, [&](float4 G) {
        cx = cx - G.x * ws;
        cy = cy - G.y * ws;
        cz = cz - G.z * ws;
    });
    float4 v = vel[i];
    v.x = v.x + cx * dt;
    v.y = v.y + cy * dt;
    v.z = v.z + cz * dt;
    vel[i] = v;
    // warm starts: the stiffness impulse this particle's solve has applied so far
    if (applied) applied[2 * (size_t)i] += own * dt;
}

template <int BLOCKS>
__global__ void __launch_bounds__(kBlock, BLOCKS) k_push(Params p, const StepConsts* __restrict__ sc, PairLists fl,
                                                 PairLists wl, const float4* __restrict__ pos,
                                                 float4* __restrict__ vel, Status* st,
                                                 float* __restrict__ applied, unsigned long long loop) {
    loop_bound(p, st, loop);
    if (__ldcg(&st->settled)) return;
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < p.n; row += gridDim.x * blockDim.x)
        push_particle(p, sc, fl, wl, fl.particle(row), row, pos, vel, applied);
}

// viscous (step.rs:229-251) + gravity of particle i (row `row` of the walk order)
__device__ __forceinline__ void viscous_particle(const Params& p, const StepConsts* __restrict__ sc,
                                                 const PairLists& fl, const PairLists& wl, uint32_t i, uint32_t row,
                                                 const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                 const float* __restrict__ rho, const float4* __restrict__ walls,
                                                 float4* __restrict__ vel_out) {
    const float dt = sc->dt;
    const float visc = sc->viscosity;
    float4 a = pos[i];
    float4 v = vel[i];
    float density = rho[i];
    float px = 0.0f, py = 0.0f, pz = 0.0f;
    each_listed2(fl, row, pos, vel, [&](uint32_t j, float g, float4 q, float4 w) {
        if (j == i) return;
        float rx = a.x - q.x, ry = a.y - q.y, rz = a.z - q.z;
        float toward = dot3(v.x - w.x, v.y - w.y, v.z - w.z, rx, ry, rz);
        if (toward < 0.0f) {
            float squeeze = toward / (dot3(rx, ry, rz, rx, ry, rz) + p.soften);
            float damp = -visc * squeeze * 2.0f / (density + w.w);  // the neighbour's density (PairRecords)
            float s = p.mass * damp;
            px = px - (rx * g) * s;
            py = py - (ry * g) * s;
            pz = pz - (rz * g) * s;
        }
    });
    float3 wv = wall_viscous(p, sc->wall_viscosity, wl, walls, row, a, v, density, TerrainDev{});
    float ax = (px + wv.x) + p.gravity.x, ay = (py + wv.y) + p.gravity.y, az = (pz + wv.z) + p.gravity.z;
    v.x = v.x + ax * dt;
    v.y = v.y + ay * dt;
    v.z = v.z + az * dt;
    vel_out[i] = v;
}

// viscous (step.rs:229-251) + gravity, velocity update (dfsph.rs:90-99); writes a new buffer
// because neighbours read the old velocities.  A row a thread in small blocks: some rows (walls,
// approaching pairs) take much longer than others, and a short block makes room as soon as its own
// are done.  Against the resident grid of 256-thread blocks, us: 57.6 -> 51.0 at 250k, 90.3 -> 83.1 at
// 500k, 152 -> 150 at 1M (64 threads: the same; the push, whose rows are alike, 70 -> 73).
__global__ void __launch_bounds__(kViscousBlock) k_viscous(Params p, const StepConsts* __restrict__ sc, PairLists fl,
                                                    PairLists wl, const float4* __restrict__ pos,
                                                    const float4* __restrict__ vel, const float* __restrict__ rho,
                                                    const float4* __restrict__ walls, float4* __restrict__ vel_out) {
    const uint32_t row = blockIdx.x * uint32_t(kViscousBlock) + threadIdx.x;
    if (row < p.n) viscous_particle(p, sc, fl, wl, fl.particle(row), row, pos, vel, rho, walls, vel_out);
}

__global__ void k_advance(Params p, const StepConsts* __restrict__ sc, const float4* __restrict__ pos_in,
                          float4* __restrict__ pos_out, float4* __restrict__ vel, Status* st,
                          float4* __restrict__ vel_pre) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = i < p.n;
    int3 nc = make_int3(0, 0, 0);
    float speed = 0.0f;
    uint32_t held = 0, bad = 0;
    if (valid) {
        float4 a = pos_in[i];
        float4 v = vel[i];
        float4 pre = v;
        uint32_t flags = 0;
        advance_one(p, sc->dt, a, v, held, bad, TerrainDev{}, &flags);
        if (vel_pre) {
            pre.w = __uint_as_float(flags);
            vel_pre[i] = pre;
        }
        pos_out[i] = a;
        vel[i] = v;
        nc = cell_of(p, a.x, a.y, a.z);
        speed = sqrtf(dot3(v.x, v.y, v.z, v.x, v.y, v.z));
        if (!(speed == speed)) speed = 0.0f;
    }
    fold_advance_stats(st, valid, nc, speed, held, bad);
}

// ---- neighbour lists on demand (mod.rs:570-606) --------------------------------------------

__global__ void k_list_count(Params p, GridDev g, const float4* __restrict__ pos, const float4* __restrict__ pts,
                             uint32_t* counts) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float4 a = pos[i];
    int3 cell = cell_of(p, a.x, a.y, a.z);
    uint32_t c = 0;
    each_near(p, g, pts, cell, a.x, a.y, a.z, [&](uint32_t, float4) { ++c; });
    counts[i] = c;
}

__global__ void k_list_fill(Params p, GridDev g, const float4* __restrict__ pos, const float4* __restrict__ pts,
                            const uint32_t* __restrict__ start, uint32_t* items) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float4 a = pos[i];
    int3 cell = cell_of(p, a.x, a.y, a.z);
    uint32_t k = start[i];
    each_near(p, g, pts, cell, a.x, a.y, a.z, [&](uint32_t j, float4) { items[k++] = j; });
}

// ---- domain (mod.rs:451-486): keep flags, then a stable compaction -------------------------

// The f32 position the readouts give: cell-relative ones rebuilt in double and rounded once.
__device__ __forceinline__ float4 absolute_of(const Params& p, const float4* __restrict__ pos,
                                              const int4* __restrict__ cells, uint32_t i) {
    float4 a = pos[i];
    if (cells) {
        int4 c = cells[i];
        const double r = p.radius;
        a.x = float(double(c.x) * r + a.x);
        a.y = float(double(c.y) * r + a.y);
        a.z = float(double(c.z) * r + a.z);
    }
    return a;
}

// drain = 0: keep what the domain holds, clamp(p) == p (mod.rs:451-486); drain = 1: keep what
// lies outside the drain box, inclusive bounds (flow.rs:154-161)
__global__ void k_domain_flags(Params p, const float4* __restrict__ pos, const int4* __restrict__ cells, float3 low,
                               float3 high, int drain, uint32_t* keep) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float4 a = absolute_of(p, pos, cells, i);
    if (drain) {
        bool inside = a.x >= low.x && a.y >= low.y && a.z >= low.z && a.x <= high.x && a.y <= high.y && a.z <= high.z;
        keep[i] = inside ? 0u : 1u;
        return;
    }
    float cx = fminf(fmaxf(a.x, low.x), high.x), cy = fminf(fmaxf(a.y, low.y), high.y),
          cz = fminf(fmaxf(a.z, low.z), high.z);
    keep[i] = (cx == a.x && cy == a.y && cz == a.z) ? 1u : 0u;
}

// ---- emitters (flow.rs:168-226) --------------------------------------------------------------
// Lattice slots of an emitter box: cnt per axis, slot (x, y, z) at index (y cnt.z + z) cnt.x + x,
// its centre low + ((x, y, z) + 1/2) spacing.  A slot is taken when a particle is nearer its
// centre than 0.9 spacing; each particle tests the 3 x 3 x 3 slots around its nearest one.

// Rust's `f as i64` (saturating, NaN to 0), then held to [-2, cells + 1]: further out reaches no slot
__device__ __forceinline__ long long nearest_slot(float v, int cells) {
    float r = roundf(v);
    long long c = (r != r) ? 0 : (r >= 9.2233720e18f ? LLONG_MAX : (r <= -9.2233720e18f ? LLONG_MIN : (long long)r));
    return c < -2 ? -2 : (c > cells + 1 ? cells + 1 : c);
}

__global__ void k_emitter_taken(Params p, const float4* __restrict__ pos, const int4* __restrict__ cells, float3 low,
                                int3 cnt, float spacing, float clear, uint32_t* __restrict__ taken) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    float4 a = absolute_of(p, pos, cells, i);
    long long nx = nearest_slot((a.x - low.x) / spacing - 0.5f, cnt.x);
    long long ny = nearest_slot((a.y - low.y) / spacing - 0.5f, cnt.y);
    long long nz = nearest_slot((a.z - low.z) / spacing - 0.5f, cnt.z);
    for (long long y = ny - 1; y <= ny + 1; ++y)
        for (long long z = nz - 1; z <= nz + 1; ++z)
            for (long long x = nx - 1; x <= nx + 1; ++x) {
                if (x < 0 || x >= cnt.x || y < 0 || y >= cnt.y || z < 0 || z >= cnt.z) continue;
                float ox = a.x - (low.x + (float(x) + 0.5f) * spacing);
                float oy = a.y - (low.y + (float(y) + 0.5f) * spacing);
                float oz = a.z - (low.z + (float(z) + 0.5f) * spacing);
                if (dot3(ox, oy, oz, ox, oy, oz) < clear) taken[(y * cnt.z + z) * cnt.x + x] = 1u;
            }
}

// After an exclusive scan of `taken` (total at taken_ex[total]): the free slots in slot order
// become particles first_id, first_id + 1, ... until `room` of them are placed.
__global__ void k_emit(uint32_t total, const uint32_t* __restrict__ taken_ex, int3 cnt, float3 low, float spacing,
                       float3 velocity, uint32_t room, uint32_t first_id, float4* __restrict__ pos_out,
                       float4* __restrict__ vel_out, uint32_t* __restrict__ ids_out, float* __restrict__ rho_out) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= total || taken_ex[s + 1] != taken_ex[s]) return;
    uint32_t rank = s - taken_ex[s];
    if (rank >= room) return;
    uint32_t x = s % uint32_t(cnt.x), z = (s / uint32_t(cnt.x)) % uint32_t(cnt.z), y = s / (uint32_t(cnt.x) * uint32_t(cnt.z));
    pos_out[rank] = make_float4(low.x + (float(x) + 0.5f) * spacing, low.y + (float(y) + 0.5f) * spacing,
                                low.z + (float(z) + 0.5f) * spacing, 0.0f);
    vel_out[rank] = make_float4(velocity.x, velocity.y, velocity.z, 0.0f);
    ids_out[rank] = first_id + rank;
    rho_out[rank] = 0.0f;
}

__global__ void k_compact(uint32_t n, const uint32_t* __restrict__ keep, const uint32_t* __restrict__ dest,
                          const uint32_t* __restrict__ ids_in, const float4* __restrict__ pos_in,
                          const float4* __restrict__ vel_in, const float* __restrict__ rho_in,
                          const int4* __restrict__ cells_in, uint32_t* __restrict__ ids_out,
                          float4* __restrict__ pos_out, float4* __restrict__ vel_out, float* __restrict__ rho_out,
                          int4* __restrict__ cells_out, const float2* __restrict__ warm_in,
                          float2* __restrict__ warm_out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !keep[i]) return;
    uint32_t f = dest[i];
    ids_out[f] = ids_in[i];
    pos_out[f] = pos_in[i];
    vel_out[f] = vel_in[i];
    rho_out[f] = rho_in[i];
    if (cells_in) cells_out[f] = cells_in[i];
    if (warm_in) warm_out[f] = warm_in[i];
}

// ---- carrying the body points through a step (couple.rs:291-318) -----------------------------

// The points at `elapsed` (start + velocity * elapsed, owner bits in start.w) and their place in
// the dense table of box (low, span): lin[i], and slot[i] among the cell's points counted so far.
__global__ void k_mover_cells(Params p, uint32_t k, const float4* __restrict__ start, const float4* __restrict__ vel,
                              float elapsed, int3 low, int3 span, uint32_t* __restrict__ lin,
                              uint32_t* __restrict__ slot, uint32_t* __restrict__ count) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= k) return;
    const float4 s0 = start[i], v = vel[i];
    const float x = s0.x + v.x * elapsed, y = s0.y + v.y * elapsed, z = s0.z + v.z * elapsed;
    const int3 c = cell_of(p, x, y, z);
    const uint32_t l = uint32_t(((long long)(c.x - low.x) * span.y + (c.y - low.y)) * span.z + (c.z - low.z));
    lin[i] = l;
    slot[i] = atomicAdd(&count[l], 1u);
}

// The points sorted by (cell, owner, place in the current order), as the host sort of
// couple.rs:291-318 orders them: a point's place in its cell is the number of the cell's points
// with a smaller (owner, current place).  Writes the sorted starts, velocities and positions at
// `elapsed` (owner bits in w).
__global__ void k_mover_order(uint32_t k, const uint32_t* __restrict__ lin, const uint32_t* __restrict__ slot,
                              const uint32_t* __restrict__ table, uint32_t* __restrict__ members,
                              const float4* __restrict__ start, const float4* __restrict__ vel, float elapsed,
                              float4* __restrict__ start_out, float4* __restrict__ vel_out,
                              float4* __restrict__ pos_out, int phase) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= k) return;
    const uint32_t l = lin[i], b = table[l];
    if (phase == 0) {  // the cell's members, in any order
        members[b + slot[i]] = i;
        return;
    }
    const uint32_t e = table[l + 1];
    const uint32_t own = __float_as_uint(start[i].w);
    uint32_t rank = 0;
    for (uint32_t q = b; q < e; ++q) {
        const uint32_t m = members[q];
        const uint32_t om = __float_as_uint(__ldg(&start[m].w));
        rank += (om < own || (om == own && m < i)) ? 1u : 0u;
    }
    const uint32_t d = b + rank;
    const float4 s0 = start[i], v = vel[i];
    start_out[d] = s0;
    vel_out[d] = v;
    pos_out[d] = make_float4(s0.x + v.x * elapsed, s0.y + v.y * elapsed, s0.z + v.z * elapsed, s0.w);
}

// k_mover_cells, the scan and both phases of k_mover_order in one block, for the few thousand points and
// cells of most scenes: the table is counted and scanned in shared memory.
constexpr int kCarryBlock = 1024;
constexpr uint32_t kCarryPoints = 16384, kCarryCells = 12000;  // 47 KB of table

__global__ void __launch_bounds__(kCarryBlock) k_mover_carry(const __grid_constant__ Params p, uint32_t k,
                                                             const float4* __restrict__ start,
                                                             const float4* __restrict__ vel, float elapsed, int3 low,
                                                             int3 span, uint32_t volume, uint32_t* lin, uint32_t* slot,
                                                             uint32_t* __restrict__ table_out, uint32_t* members,
                                                             float4* __restrict__ start_out, float4* __restrict__ vel_out,
                                                             float4* __restrict__ pos_out) {
    extern __shared__ uint32_t table[];  // volume words
    __shared__ uint32_t warp_sums[kCarryBlock / 32];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    for (uint32_t c = t; c < volume; c += kCarryBlock) table[c] = 0u;
    __syncthreads();
    for (uint32_t i = t; i < k; i += kCarryBlock) {
        const float4 s0 = start[i], v = vel[i];
        const float x = s0.x + v.x * elapsed, y = s0.y + v.y * elapsed, z = s0.z + v.z * elapsed;
        const int3 c = cell_of(p, x, y, z);
        const uint32_t l = uint32_t(((long long)(c.x - low.x) * span.y + (c.y - low.y)) * span.z + (c.z - low.z));
        lin[i] = l;
        slot[i] = atomicAdd(&table[l], 1u);
    }
    __syncthreads();
    // exclusive scan: a run of cells a thread
    const uint32_t per = (volume + kCarryBlock - 1) / kCarryBlock, c0 = min(t * per, volume), c1 = min(c0 + per, volume);
    uint32_t sum = 0;
    for (uint32_t c = c0; c < c1; ++c) sum += table[c];
    uint32_t upto = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t other = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= uint32_t(d)) upto += other;
    }
    if (lane == 31) warp_sums[warp] = upto;
    __syncthreads();
    uint32_t at = upto - sum;
    for (uint32_t w = 0; w < warp; ++w) at += warp_sums[w];
    for (uint32_t c = c0; c < c1; ++c) {
        const uint32_t here = table[c];
        table[c] = at;
        table_out[c] = at;
        at += here;
    }
    if (t == 0) table_out[volume] = k;
    __syncthreads();
    for (uint32_t i = t; i < k; i += kCarryBlock) members[table[lin[i]] + slot[i]] = i;
    __syncthreads();
    for (uint32_t i = t; i < k; i += kCarryBlock) {
        const uint32_t l = lin[i], b = table[l], e = l + 1u < volume ? table[l + 1u] : k;
        const float4 s0 = start[i], v = vel[i];
        const uint32_t own = __float_as_uint(s0.w);
        uint32_t rank = 0;
        for (uint32_t q = b; q < e; ++q) {
            const uint32_t m = members[q], om = __float_as_uint(__ldg(&start[m].w));
            rank += (om < own || (om == own && m < i)) ? 1u : 0u;
        }
        const uint32_t d = b + rank;
        start_out[d] = s0;
        vel_out[d] = v;
        pos_out[d] = make_float4(s0.x + v.x * elapsed, s0.y + v.y * elapsed, s0.z + v.z * elapsed, s0.w);
    }
}

// ---- the particles a coupled body's lift reads (lift.rs:29-60) -----------------------------------

// keep[i] = 1 for a particle inside any of the boxes (low, high pairs, bounds inclusive, NaN
// bounds ignored and NaN positions outside, as the host's clamp test min(max(p, low), high) == p)
__global__ void k_in_boxes(uint32_t n, const float4* __restrict__ pos, const float3* __restrict__ boxes,
                           uint32_t count, uint32_t* __restrict__ keep) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = pos[i];
    uint32_t in = 0;
    if (a.x == a.x && a.y == a.y && a.z == a.z) {
        for (uint32_t b = 0; b < count && !in; ++b) {
            const float3 lo = boxes[2 * b], hi = boxes[2 * b + 1];
            in = !(lo.x > a.x) && !(a.x > hi.x) && !(lo.y > a.y) && !(a.y > hi.y) && !(lo.z > a.z) && !(a.z > hi.z);
        }
    }
    keep[i] = in;
}

// the kept particles in index order: their index, position and velocity (xyz, 6 floats)
__global__ void k_gather_kept(uint32_t n, const uint32_t* __restrict__ keep, const uint32_t* __restrict__ at,
                              const float4* __restrict__ pos, const float4* __restrict__ vel,
                              uint32_t* __restrict__ index, float* __restrict__ pv) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !keep[i]) return;
    const uint32_t k = at[i];
    const float4 a = pos[i], v = vel[i];
    index[k] = i;
    float* o = pv + 6 * size_t(k);
    o[0] = a.x;
    o[1] = a.y;
    o[2] = a.z;
    o[3] = v.x;
    o[4] = v.y;
    o[5] = v.z;
}

// vel[index[k]].xyz = v3[k]
__global__ void k_scatter_velocities(uint32_t m, const uint32_t* __restrict__ index, const float* __restrict__ v3,
                                     float4* __restrict__ vel) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    const uint32_t i = index[k];
    vel[i] = make_float4(v3[3 * size_t(k)], v3[3 * size_t(k) + 1], v3[3 * size_t(k) + 2], 0.0f);
}

__global__ void k_set_consts(StepConsts c, StepConsts* out) { *out = c; }

// xyz triples <-> float4, so host copies move 12 bytes a particle
__global__ void k_pack3(uint32_t n, const float4* __restrict__ in, float* __restrict__ out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = in[i];
    out[3 * i] = v.x;
    out[3 * i + 1] = v.y;
    out[3 * i + 2] = v.z;
}

// xyz triples into float4 slots; `bad` (optional) counts triples with a non finite component
__global__ void k_unpack3(uint32_t n, const float* __restrict__ in, float4* __restrict__ out, uint32_t* bad) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x = in[3 * i], y = in[3 * i + 1], z = in[3 * i + 2];
    if (bad && !(isfinite(x) && isfinite(y) && isfinite(z))) atomicAdd(bad, 1u);
    out[i] = make_float4(x, y, z, 0.0f);
}

// A whole state in one pass, in: n position triples, then n velocity triples; with the cell box, the
// fastest speed and whether a component is non finite in the status.  Two unpacks and a pass over
// what they wrote took two launches and 32 bytes a particle more: with the one pack a pass of four 8k
// steps 435 -> 426 us, of two 315k steps 851 -> 843.
__global__ void k_unpack_state(Params p, const float* __restrict__ in, float4* __restrict__ pos,
                               float4* __restrict__ vel, Status* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < p.n;
    int3 c = make_int3(0, 0, 0);
    float speed = 0.0f;
    uint32_t bad = 0;
    if (valid) {
        const size_t a = 3 * size_t(i), b = 3 * (size_t(p.n) + i);
        const float x = in[a], y = in[a + 1], z = in[a + 2], vx = in[b], vy = in[b + 1], vz = in[b + 2];
        bad = isfinite(x) && isfinite(y) && isfinite(z) && isfinite(vx) && isfinite(vy) && isfinite(vz) ? 0u : 1u;
        pos[i] = make_float4(x, y, z, 0.0f);
        vel[i] = make_float4(vx, vy, vz, 0.0f);
        c = cell_of(p, x, y, z);
        speed = sqrtf(dot3(vx, vy, vz, vx, vy, vz));  // Vec3::length, as k_state_stats
        if (!(speed == speed)) speed = 0.0f;
    }
    fold_advance_stats(st, valid, c, speed, 0u, bad);
}

// a whole state back into n position triples and n velocity triples
__global__ void k_pack_state(uint32_t n, const float4* __restrict__ pos, const float4* __restrict__ vel,
                             float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t a = 3 * size_t(i), b = 3 * (size_t(n) + i);
    const float4 x = pos[i], v = vel[i];
    out[a] = x.x;
    out[a + 1] = x.y;
    out[a + 2] = x.z;
    out[b] = v.x;
    out[b + 1] = v.y;
    out[b + 2] = v.z;
}

// ---- launchers ------------------------------------------------------------------------------

static std::atomic<uint64_t> g_launches{0};
uint64_t kernel_launches() { return g_launches.load(); }
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
void note_launches(int64_t k) { g_launches.fetch_add(uint64_t(k), std::memory_order_relaxed); }

static inline uint32_t blocks_for(uint32_t n) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return (n + kBlock - 1) / kBlock;
}

// The list passes' grids (the solves' check and push, the density pass, the WCSPH force): with
// SLF_SOLVER_RESIDENT, no more blocks than the SMs hold at once (each block then strides over
// rows), so no launch ends on a partial wave and the check's residual sums fewer block partials.
#ifndef SLF_SOLVER_RESIDENT
#define SLF_SOLVER_RESIDENT 1
#endif
// resident blocks of k_rate<0>, k_rate<1> and k_push (as large grids run them), k_density<0>,
// k_density<1> and k_wcsph_force on the device (prepare_solver_grids; 0: not known yet, the grid then covers every row)
static std::atomic<uint32_t> g_resident[6] = {0, 0, 0, 0, 0, 0};

// blocks of the density pass up to which it runs wide: two a SM
static std::atomic<uint32_t> g_wide_blocks{0};
// blocks of the check and the push up to which no SM holds more than kFewBlocks
static std::atomic<uint32_t> g_few_blocks{0};

void prepare_solver_grids() {
    if (!SLF_SOLVER_RESIDENT || g_resident[2].load()) return;
    int dev = 0, sms = 0, per[6] = {0, 0, 0, 0, 0, 0};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[0], k_rate<0, kRateBlocks>, kBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[1], k_rate<1, kRateBlocks>, kBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[2], k_push<kPushBlocks>, kBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[3], k_density<0, true, false>, kBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[4], k_density<1, false, false>, kBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[5], k_wcsph_force<true>, kBlock, 0);
    g_wide_blocks.store(2u * uint32_t(std::max(sms, 0)));
    g_few_blocks.store(uint32_t(kFewBlocks * std::max(sms, 0)));
    for (int k = 0; k < 6; ++k) g_resident[k].store(uint32_t(std::max(per[k], 0) * std::max(sms, 0)));
}

static uint32_t solver_blocks(uint32_t n, int kernel) {
    uint32_t nb = blocks_for(n);
    uint32_t resident = g_resident[kernel].load();
    return resident && resident < nb ? resident : nb;
}

void launch_pack3(uint32_t n, const float4* in, float* out, cudaStream_t s) {
    if (n) k_pack3<<<blocks_for(n), kBlock, 0, s>>>(n, in, out);
}

void launch_unpack_state(const Params& p, const float* in, float4* pos, float4* vel, Status* st, cudaStream_t s) {
    if (p.n) k_unpack_state<<<blocks_for(p.n), kBlock, 0, s>>>(p, in, pos, vel, st);
}

void launch_pack_state(uint32_t n, const float4* pos, const float4* vel, float* out, cudaStream_t s) {
    if (n) k_pack_state<<<blocks_for(n), kBlock, 0, s>>>(n, pos, vel, out);
}

void launch_unpack3(uint32_t n, const float* in, float4* out, cudaStream_t s, uint32_t* bad) {
    if (n) k_unpack3<<<blocks_for(n), kBlock, 0, s>>>(n, in, out, bad);
}

void launch_state_stats(const Params& p, const float4* pos, const float4* vel, Status* st, cudaStream_t s) {
    if (p.n) k_state_stats<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos, vel, st);
}

void launch_max_compression(const Params& p, const float* rho, Status* st, cudaStream_t s) {
    if (p.n) k_max_compression<<<blocks_for(p.n), kBlock, 0, s>>>(p, rho, st);
}

void launch_post_status(const Status* st, Status* out, uint32_t* posted, cudaStream_t s, uint32_t cap,
                        uint32_t* spoiled) {
    note_launch();
    k_post_status<<<1, 32, 0, s>>>(st, out, posted, cap, spoiled);
}

void launch_count_cells(const Params& p, const float4* pos, const int4* cells, int3 low, int3 span, uint32_t* count,
                        uint32_t* lin, uint32_t* slot, cudaStream_t s, SubstepBegin begin) {
    if (p.n) k_count_cells<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos, cells, low, span, count, lin, slot, begin);
}

void launch_grid_near(const GridDev& g, uint32_t* near, cudaStream_t s) {
    const uint32_t volume = uint32_t(g.sx) * uint32_t(g.sy) * uint32_t(g.sz);
    if (g.mode == 1 && volume) k_grid_near<<<blocks_for(volume), kBlock, 0, s>>>(g, near);
}

size_t scan_tiles(uint32_t m) { return (m + kScanTile - 1) / kScanTile; }

void launch_exclusive_scan(uint32_t* data, uint32_t m, uint32_t* tile_sums, cudaStream_t s) {
    if (m == 0) return;
    const uint32_t tiles = (uint32_t)scan_tiles(m);
    const int wide = (reinterpret_cast<uintptr_t>(data) & 15u) == 0;
    k_scan_tiles<<<tiles, kBlock, 0, s>>>(data, m, tile_sums, wide);
    g_launches.fetch_add(tiles == 1 ? 1 : tiles <= kScanOwnSums ? 2 : 3, std::memory_order_relaxed);
    if (tiles == 1) return;
    if (tiles <= kScanOwnSums) {
        k_scan_finish<<<tiles, kBlock, 0, s>>>(data, m, tile_sums, wide);
        return;
    }
    k_scan_sums<<<1, kBlock, 0, s>>>(tile_sums, tiles);
    k_scan_add<<<tiles, kBlock, 0, s>>>(data, m, tile_sums);
}

void launch_scatter_members(uint32_t n, const uint32_t* lin, const uint32_t* slot, const uint32_t* start,
                            const uint32_t* ids, uint32_t* members, cudaStream_t s) {
    if (n) k_scatter_members<<<blocks_for(n), kBlock, 0, s>>>(n, lin, slot, start, ids, members);
}

void launch_rank_reorder(uint32_t n, const uint32_t* lin, const uint32_t* start, const uint32_t* members,
                         const uint32_t* ids_in, const float4* pos_in, const float4* vel_in, const float* rho_in,
                         const int4* cells_in, uint32_t* ids_out, float4* pos_out, float4* vel_out, float* rho_out,
                         int4* cells_out, const float2* warm_in, float2* warm_out, uint32_t skip_begin,
                         uint32_t skip_end, Status* st, uint32_t* dest, int3 span, int pad, uint32_t* order,
                         cudaStream_t s) {
    if (n)
        k_rank_reorder<<<blocks_for(n), kBlock, 0, s>>>(n, lin, start, members, ids_in, pos_in, vel_in, rho_in,
                                                        cells_in, ids_out, pos_out, vel_out, rho_out, cells_out,
                                                        warm_in, warm_out,
                                                        skip_begin, skip_end, st, dest, span, pad, order);
}

// blocks of a pass that gives each row `lanes` lanes
static uint32_t group_blocks(uint32_t n, int lanes) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    const uint32_t rows = uint32_t(kGroupBlock / lanes);
    return (n + rows - 1) / rows;
}

size_t density_scratch_rows(uint32_t n, float support, bool dfsph) {
    static_assert(kDensityRowsMin == kBlock, "a block's rows");
    // one a thread of the density pass's grid
    const uint32_t nb = (n + kBlock - 1) / kBlock, r0 = g_resident[3].load(), r1 = g_resident[4].load();
    const uint32_t resident = r0 && r1 ? std::max(r0, r1) : nb;
    // (with lanes to share, one a row of the grid, whose last tile may be part empty)
    const size_t group = group_lanes(n, support, dfsph) ? size_t(n + kGroupBlock) : 0;
    return std::max(size_t(std::min(resident, nb)) * kBlock, group);
}

void launch_density(const Params& p, const GridDev& fg, const GridDev& wg, float4* pos, const float4* walls,
                    const PairLists& fl, const PairLists& wl, float* rho, float* press, float* scaled, float* alpha,
                    Status* st, const TerrainDev& T, float4* slope, cudaStream_t s, const MoverDev& M,
                    uint32_t* scratch, size_t scratch_rows, float4* vel) {
    if (!p.n) return;
    const PairRecords rec{reinterpret_cast<float*>(pos), reinterpret_cast<float*>(vel)};
    const DensityIn in{{fg, wg}, {pos, walls}, {fl, wl}};
    // (terrain, whose sites every lane would take alike, and a DFSPH row's body points keep a thread a row)
    const bool shared = T.regions == 0 && slope == nullptr && (p.solver == 0 || M.count == 0) &&
                        scratch_rows >= size_t(p.n) + kGroupBlock;
    if (shared && with_lanes(group_lanes(p.n, p.radius / p.spacing, p.solver != 0), [&](auto lanes) {
            constexpr int L = decltype(lanes)::value;
            const uint32_t nb = group_blocks(p.n, L);
            auto launch = [&](auto flight) {
                constexpr int F = decltype(flight)::value;
                if (p.solver != 0)
                    k_density_group<1, false, L, F><<<nb, kGroupBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, M,
                                                                               scratch, rec);
                else if (M.count)
                    k_density_group<0, true, L, F><<<nb, kGroupBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, M,
                                                                              scratch, rec);
                else
                    k_density_group<0, false, L, F><<<nb, kGroupBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, M,
                                                                               scratch, rec);
            };
            // a cell's points at rest: few enough of them, L lanes test the 27 cells end to end (216
            // candidates at support 2, L = 32, 1000 particles: 27 -> 15 us against a cell at a time);
            // many, and a lane keeps four of a cell's in flight (64 at support 4, L = 4, 74k
            // particles: 293 -> 273 us against two, at support 2 73 -> 90)
            const float support = p.radius / p.spacing, points = support * support * support;
            if constexpr (L >= 8) {
                if (points <= 2.0f * L) return launch(std::integral_constant<int, 0>{});
            }
            if (points < 16.0f) launch(std::integral_constant<int, 2>{});
            else launch(std::integral_constant<int, 4>{});
        }))
        return;
    const uint32_t nb = uint32_t(std::min<size_t>(solver_blocks(p.n, p.solver == 0 ? 3 : 4), scratch_rows / kBlock));
    auto launch = [&](auto wide) {
        constexpr bool W = decltype(wide)::value;
        // (no DFSPH step takes terrain, but the densities of a DFSPH world on terrain have its ground)
        const bool extra = T.regions || M.count || slope;
        if (p.solver != 0 && extra)
            k_density<1, true, W><<<nb, kBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, T, slope, M, scratch, rec);
        else if (p.solver != 0)
            k_density<1, false, W><<<nb, kBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, T, slope, M, scratch, rec);
        else if (extra)
            k_density<0, true, W><<<nb, kBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, T, slope, M, scratch, rec);
        else
            k_density<0, false, W><<<nb, kBlock, 0, s>>>(p, in, rho, press, scaled, alpha, st, T, slope, M, scratch, rec);
    };
    if (nb <= g_wide_blocks.load()) launch(std::true_type{});
    else launch(std::false_type{});
}

void launch_wcsph_force(const Params& p, const StepConsts* sc, const PairLists& fl, const PairLists& wl,
                        const float4* pos, const float4* vel, const float* rho, const float* press,
                        const float* scaled, const float4* walls, float4* pos_out, float4* vel_out, Status* st,
                        float4* vel_pre, const TerrainDev& T, const float4* slope, cudaStream_t s,
                        const MoverDev& M) {
    if (!p.n) return;
    if (T.regions == 0 && slope == nullptr && with_lanes(group_lanes(p.n, p.radius / p.spacing, false), [&](auto lanes) {
            constexpr int L = decltype(lanes)::value;
            const uint32_t nb = group_blocks(p.n, L);
            if (M.count)
                k_wcsph_force_group<true, L><<<nb, kGroupBlock, 0, s>>>(p, sc, fl, wl, pos, vel, rho, press, scaled,
                                                                        walls, pos_out, vel_out, st, vel_pre, M);
            else
                k_wcsph_force_group<false, L><<<nb, kGroupBlock, 0, s>>>(p, sc, fl, wl, pos, vel, rho, press, scaled,
                                                                         walls, pos_out, vel_out, st, vel_pre, M);
        }))
        return;
    const uint32_t nb = solver_blocks(p.n, 5);
    if (T.regions || M.count || slope)
        k_wcsph_force<true><<<nb, kBlock, 0, s>>>(p, sc, fl, wl, pos, vel, rho, press, scaled, walls, pos_out, vel_out,
                                                  st, vel_pre, T, slope, M);
    else
        k_wcsph_force<false><<<nb, kBlock, 0, s>>>(p, sc, fl, wl, pos, vel, rho, press, scaled, walls, pos_out, vel_out,
                                                   st, vel_pre, T, slope, M);
}

void launch_mover_felt(const Params& p, float mover_damping, const MoverDev& M, const float4* pos, const float4* vel,
                       const float* rho, const float* press, const float* scaled, const float4* centre, float elapsed,
                       uint32_t bodies, float4* felt, cudaStream_t s) {
    if (!p.n) return;
    static_assert(kFeltBlock == 512, "a block a chunk, a thread a particle");
    k_mover_felt<<<(p.n + 511u) / 512u, kFeltBlock, 0, s>>>(p, mover_damping, M, pos, vel, rho, press, scaled, centre, elapsed,
                                                            bodies, felt);
    note_launch();
}

// What each body took this substep, folded into its step's impulse as the host folds it
// (step.rs:173-221): chunk by chunk in order, impulse + force * dt, angular + torque * dt.  A block
// a body: its threads bring the chunks' records into shared memory 256 at a time and one thread
// adds them in order.
// A substep that will run again or fails (its lists outgrew cap, or it left non-finite values) adds
// nothing: its chunks are queued before the host has read its status.
__global__ void k_mover_fold(uint32_t chunks, uint32_t bodies, const float4* __restrict__ felt, float dt,
                             float4* __restrict__ impulse, const uint32_t* __restrict__ spoiled) {
    if (*spoiled) return;
    __shared__ float4 force[kBlock], torque[kBlock];
    const uint32_t b = blockIdx.x, t = threadIdx.x;
    float4 imp = impulse[2 * size_t(b)], ang = impulse[2 * size_t(b) + 1];
    for (uint32_t base = 0; base < chunks; base += kBlock) {
        const uint32_t c = base + t;
        if (c < chunks) {
            force[t] = felt[2 * (size_t(c) * bodies + b)];
            torque[t] = felt[2 * (size_t(c) * bodies + b) + 1];
        }
        __syncthreads();
        if (t == 0) {
            const uint32_t here = chunks - base < uint32_t(kBlock) ? chunks - base : uint32_t(kBlock);
#pragma unroll 8
            for (uint32_t j = 0; j < here; ++j) {
                const float4 f = force[j], q = torque[j];
                imp = make_float4(imp.x + f.x * dt, imp.y + f.y * dt, imp.z + f.z * dt, 0.0f);
                ang = make_float4(ang.x + q.x * dt, ang.y + q.y * dt, ang.z + q.z * dt, 0.0f);
            }
        }
        __syncthreads();
    }
    if (t == 0) {
        impulse[2 * size_t(b)] = imp;
        impulse[2 * size_t(b) + 1] = ang;
    }
}

void launch_mover_fold(uint32_t n, uint32_t bodies, const float4* felt, float dt, float4* impulse,
                       const uint32_t* spoiled, cudaStream_t s) {
    if (!n || !bodies) return;
    k_mover_fold<<<bodies, kBlock, 0, s>>>((n + 511u) / 512u, bodies, felt, dt, impulse, spoiled);
    note_launch();
}

void launch_cells_wet(const GridDev& g, int3 lo, int3 hi, uint32_t* wet, cudaStream_t s) {
    long long total = ((long long)hi.x - lo.x + 1) * ((long long)hi.y - lo.y + 1) * ((long long)hi.z - lo.z + 1);
    if (total <= 0) return;
    long long blocks = std::min<long long>((total + kBlock - 1) / kBlock, 4096);
    k_cells_wet<<<uint32_t(blocks), kBlock, 0, s>>>(g, lo, hi, wet);
    note_launch();
}

size_t rate_partial_bytes(uint32_t n) { return (n + kBlock - 1) / kBlock * (sizeof(DD) + sizeof(uint32_t)) + 64; }


void launch_rate(int which, const Params& p, const StepConsts* sc, const PairLists& fl, const PairLists& wl,
                 float4* pos, const float4* vel, const float* rho, const float* alpha, void* partials,
                 Status* st, SolveRec rec, cudaStream_t s, unsigned long long loop) {
    if (!p.n) return;
    // the partials' room is for one block a 256 rows; the grid takes at most that many
    uint32_t nb = solver_blocks(p.n, which == 0 ? 0 : 1);
    DD* part = static_cast<DD*>(partials);
    uint32_t* loaded = reinterpret_cast<uint32_t*>(part + (p.n + kBlock - 1) / kBlock);
    auto launch = [&](auto w, auto few) {
        k_rate<decltype(w)::value, decltype(few)::value><<<nb, kBlock, 0, s>>>(
            p, sc, fl, wl, pos, vel, rho, alpha, reinterpret_cast<float*>(pos), part, loaded, st, rec, loop);
    };
    auto sized = [&](auto w) {
        if (nb <= g_few_blocks.load()) launch(w, std::integral_constant<int, kFewBlocks>{});
        else launch(w, std::integral_constant<int, kRateBlocks>{});
    };
    if (which == 0) sized(std::integral_constant<int, 0>{});
    else sized(std::integral_constant<int, 1>{});
}

void launch_push(const Params& p, const StepConsts* sc, const PairLists& fl, const PairLists& wl, const float4* pos,
                 float4* vel, Status* st, float* applied, cudaStream_t s, unsigned long long loop) {
    if (!p.n) return;
    const uint32_t nb = solver_blocks(p.n, 2);
    if (nb <= g_few_blocks.load()) k_push<kFewBlocks><<<nb, kBlock, 0, s>>>(p, sc, fl, wl, pos, vel, st, applied, loop);
    else k_push<kPushBlocks><<<nb, kBlock, 0, s>>>(p, sc, fl, wl, pos, vel, st, applied, loop);
}

// Warm start of a solve: the stiffness that applies `share` of the impulse S the particle's last
// solve of this kind applied (S = sum of kappa dt), at this substep's dt, into the position's
// spare lane for one push; S restarts from that push's impulse.
__global__ void k_warm_kappa(Params p, const StepConsts* __restrict__ sc, float share, float* __restrict__ applied,
                             float4* __restrict__ pos) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float dt = sc->dt;
    const float impulse = share * applied[2 * (size_t)i];
    float kappa = impulse != 0.0f ? impulse / dt : impulse;
    pos[i].w = kappa;
    applied[2 * (size_t)i] = kappa * dt;
}

void launch_warm_kappa(const Params& p, const StepConsts* sc, float share, float* applied, float4* pos, cudaStream_t s) {
    if (p.n) k_warm_kappa<<<blocks_for(p.n), kBlock, 0, s>>>(p, sc, share, applied, pos);
}

void launch_viscous(const Params& p, const StepConsts* sc, const PairLists& fl, const PairLists& wl, const float4* pos,
                    const float4* vel, const float* rho, const float4* walls, float4* vel_out, cudaStream_t s) {
    if (!p.n) return;
    note_launch();
    k_viscous<<<(p.n + kViscousBlock - 1) / kViscousBlock, kViscousBlock, 0, s>>>(p, sc, fl, wl, pos, vel, rho, walls,
                                                                                  vel_out);
}

void launch_advance(const Params& p, const StepConsts* sc, const float4* pos_in, float4* pos_out, float4* vel,
                    Status* st, float4* vel_pre, cudaStream_t s) {
    if (p.n) k_advance<<<blocks_for(p.n), kBlock, 0, s>>>(p, sc, pos_in, pos_out, vel, st, vel_pre);
}

void launch_list_count(const Params& p, const GridDev& g, const float4* pos, const float4* pts, uint32_t* counts,
                       cudaStream_t s) {
    if (p.n) k_list_count<<<blocks_for(p.n), kBlock, 0, s>>>(p, g, pos, pts, counts);
}

void launch_list_fill(const Params& p, const GridDev& g, const float4* pos, const float4* pts, const uint32_t* start,
                      uint32_t* items, cudaStream_t s) {
    if (p.n) k_list_fill<<<blocks_for(p.n), kBlock, 0, s>>>(p, g, pos, pts, start, items);
}

void launch_emitter_taken(const Params& p, const float4* pos, const int4* cells, float3 low, int3 cnt, float spacing,
                          float clear, uint32_t* taken, cudaStream_t s) {
    if (p.n) k_emitter_taken<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos, cells, low, cnt, spacing, clear, taken);
}

void launch_emit(uint32_t total, const uint32_t* taken_ex, int3 cnt, float3 low, float spacing, float3 velocity,
                 uint32_t room, uint32_t first_id, float4* pos_out, float4* vel_out, uint32_t* ids_out, float* rho_out,
                 cudaStream_t s) {
    if (total && room)
        k_emit<<<blocks_for(total), kBlock, 0, s>>>(total, taken_ex, cnt, low, spacing, velocity, room, first_id, pos_out,
                                                    vel_out, ids_out, rho_out);
}

void launch_carry_movers(const Params& p, uint32_t k, const float4* start, const float4* vel, float elapsed, int3 low,
                         int3 span, uint32_t volume, uint32_t* lin, uint32_t* slot, uint32_t* table, uint32_t* tiles,
                         uint32_t* members, float4* start_out, float4* vel_out, float4* pos_out, cudaStream_t s) {
    if (!k) return;
    if (k <= kCarryPoints && volume <= kCarryCells) {
        k_mover_carry<<<1, kCarryBlock, volume * 4, s>>>(p, k, start, vel, elapsed, low, span, volume, lin, slot, table,
                                                         members, start_out, vel_out, pos_out);
        note_launch();
        return;
    }
    cudaMemsetAsync(table, 0, (size_t(volume) + 1) * 4, s);
    k_mover_cells<<<blocks_for(k), kBlock, 0, s>>>(p, k, start, vel, elapsed, low, span, lin, slot, table);
    launch_exclusive_scan(table, volume, tiles, s);
    k_mover_order<<<blocks_for(k), kBlock, 0, s>>>(k, lin, slot, table, members, start, vel, elapsed, start_out,
                                                   vel_out, pos_out, 0);
    k_mover_order<<<blocks_for(k), kBlock, 0, s>>>(k, lin, slot, table, members, start, vel, elapsed, start_out,
                                                   vel_out, pos_out, 1);
    g_launches.fetch_add(3, std::memory_order_relaxed);
}

void launch_in_boxes(uint32_t n, const float4* pos, const float3* boxes, uint32_t count, uint32_t* keep, cudaStream_t s) {
    if (n) k_in_boxes<<<blocks_for(n), kBlock, 0, s>>>(n, pos, boxes, count, keep);
}

void launch_gather_kept(uint32_t n, const uint32_t* keep, const uint32_t* at, const float4* pos, const float4* vel,
                        uint32_t* index, float* pv, cudaStream_t s) {
    if (n) k_gather_kept<<<blocks_for(n), kBlock, 0, s>>>(n, keep, at, pos, vel, index, pv);
}

void launch_scatter_velocities(uint32_t m, const uint32_t* index, const float* v3, float4* vel, cudaStream_t s) {
    if (m) k_scatter_velocities<<<blocks_for(m), kBlock, 0, s>>>(m, index, v3, vel);
}

void launch_domain_flags(const Params& p, const float4* pos, const int4* cells, float3 low, float3 high, int drain,
                         uint32_t* keep, cudaStream_t s) {
    if (p.n) k_domain_flags<<<blocks_for(p.n), kBlock, 0, s>>>(p, pos, cells, low, high, drain, keep);
}

void launch_compact(uint32_t n, const uint32_t* keep, const uint32_t* dest, const uint32_t* ids_in,
                    const float4* pos_in, const float4* vel_in, const float* rho_in, const int4* cells_in,
                    uint32_t* ids_out, float4* pos_out, float4* vel_out, float* rho_out, int4* cells_out,
                    const float2* warm_in, float2* warm_out, cudaStream_t s) {
    if (n)
        k_compact<<<blocks_for(n), kBlock, 0, s>>>(n, keep, dest, ids_in, pos_in, vel_in, rho_in, cells_in, ids_out,
                                                   pos_out, vel_out, rho_out, cells_out, warm_in, warm_out);
}

void launch_set_consts(const StepConsts& c, StepConsts* out, cudaStream_t s) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    k_set_consts<<<1, 1, 0, s>>>(c, out);
}

}  // namespace slf
