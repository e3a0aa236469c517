// scan.cuh -- the density pass's candidate scan, shared by the exact and the fast kernels.
#pragma once

#include "fluid_device.cuh"

namespace slf {

// Lists the points of cells [b, e) within reach of `at`, in array order: each kept index goes to
// out[nf * 32] (room for `cap`; the count goes on past it).  Four candidates' gathers are in flight
// at a time, and a kept one costs a predicated store and an add: no branch, so the lanes of a warp
// that keep nothing do not wait for those that do.  axy, az: the negated position; x and y of the
// test run packed, each operation rounded on its own whatever the compiler's contraction setting, as
// each_in_cell's.  REL: positions are offsets from their cells' corners, sxy and sz the step to this
// cell in metres, and a kept index takes the bits `code` (the step, encode_entry).
template <int kScanUnroll, bool REL>
__device__ __forceinline__ void scan_range(const Params& p, const float4* __restrict__ pts, uint32_t b, uint32_t e,
                                           f32x2 axy, float az, uint32_t* out, uint32_t cap, uint32_t& nf, f32x2 sxy,
                                           float sz, uint32_t code) {
    const ulonglong2* __restrict__ q2 = reinterpret_cast<const ulonglong2*>(pts);
#pragma unroll 1
    for (uint32_t j = b; j < e; j += kScanUnroll) {
        ulonglong2 q[kScanUnroll];
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            if (j + u < e) q[u] = __ldg(q2 + j + u);
        }
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            f32x2 oxy = add2(f32x2{q[u].x}, axy);
            float oz = __fadd_rn(__uint_as_float(uint32_t(q[u].y)), az);
            if (REL) oxy = add2(oxy, sxy), oz = __fadd_rn(oz, sz);
            float x2, y2;
            unpack2(mul2(oxy, oxy), x2, y2);
            const bool keep = j + u < e && __fadd_rn(__fadd_rn(x2, y2), __fmul_rn(oz, oz)) < p.reach;
            if (keep && nf < cap) out[size_t(nf) * 32u] = (j + u) | code;
            nf += keep ? 1u : 0u;
        }
    }
}

// The scan through tables that need bounds checks or a search, out of line: what it would hold in
// registers stays out of the density pass.
static __device__ __noinline__ uint32_t scan_checked(const Params& p, const GridDev& g, const float4* __restrict__ pts,
                                              int3 cell, float x, float y, float z, uint32_t* out,
                                              uint32_t cap, uint32_t stride) {
    uint32_t nf = 0;
    each_near(p, g, pts, cell, x, y, z, [&](uint32_t j, float4) {
        if (nf < cap) out[size_t(nf) * stride] = j;
        ++nf;
    });
    return nf;
}

// Lists the points of `g` within reach of (x, y, z) in the reference's list order (each_near's).
// Where the table knows which of a cell's 27 cells hold points (GridDev::near, the walls), only those
// are visited; a cell with its 26 neighbours inside a dense table needs no bounds checks (the world
// pads the fluid's table so that every particle's has).
// Checked (optional): the scan that tables with checks take instead of scan_checked.
struct ScanChecked {
    __device__ __forceinline__ uint32_t operator()(const Params& p, const GridDev& g, const float4* __restrict__ pts,
                                                   int3 cell, float x, float y, float z, uint32_t* out,
                                                   uint32_t cap) const {
        return scan_checked(p, g, pts, cell, x, y, z, out, cap, 32u);
    }
};
template <int kScanUnroll, bool REL = false, class Checked = ScanChecked>
__device__ __forceinline__ uint32_t scan_near(const Params& p, const GridDev& g, const float4* __restrict__ pts,
                                              int3 cell, float x, float y, float z, uint32_t* out,
                                              uint32_t cap, Checked&& checked = Checked{}) {
    if (g.mode == 0) return 0u;
    const long long bx = (long long)cell.x - g.lx, by = (long long)cell.y - g.ly, bz = (long long)cell.z - g.lz;
    const int edge = g.near ? 0 : 1;  // cells that a walk without checks keeps away from the box's faces
    if (g.mode != 1 || bx < edge || bx + edge >= g.sx || by < edge || by + edge >= g.sy || bz < edge ||
        bz + edge >= g.sz)
        return checked(p, g, pts, cell, x, y, z, out, cap);
    const f32x2 axy = pack2(-x, -y);
    const float az = -z;
    const uint32_t slab = uint32_t(g.sy) * uint32_t(g.sz);
    const uint32_t c0 = (uint32_t(bx) * uint32_t(g.sy) + uint32_t(by)) * uint32_t(g.sz) + uint32_t(bz);
    uint32_t nf = 0;
#pragma unroll 1
    for (uint32_t mask = g.near ? __ldg(&g.near[c0]) : (1u << 27) - 1u; mask; mask &= mask - 1u) {
        const int t = __ffs(int(mask)) - 1;
        const int dx = t % 3 - 1, dy = t / 3 % 3 - 1, dz = t / 9 - 1;
        const uint32_t c = c0 + uint32_t(dx * int(slab) + dy * g.sz + dz);
        // (the step's products are exact, and its code is encode_entry's)
        scan_range<kScanUnroll, REL>(p, pts, __ldg(&g.start[c]), __ldg(&g.start[c + 1]), axy, az, out, cap, nf,
                                     REL ? pack2(float(dx) * p.radius, float(dy) * p.radius) : axy,
                                     float(dz) * p.radius,
                                     REL ? uint32_t((dx + 1) | ((dy + 1) << 2) | ((dz + 1) << 4)) << 26 : 0u);
    }
    return nf;
}

}  // namespace slf
