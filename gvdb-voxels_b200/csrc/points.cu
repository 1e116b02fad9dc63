// points.cu -- point insertion and binning.
//
//   InsertPoints (V:5219-5267, P:19-36, P:59-72): per point the leaf it
//     falls in (pnode), its slot inside that leaf (poff) and per-leaf
//     counts (gcnt); with `prefix`, a counting sort of positions by leaf.
//   Kernel-splat binning (no reference counterpart): a
//     counting sort of points by (atlas slot, region) where the 27 regions
//     say which neighbouring bricks a point's stencil reaches; the splat
//     kernels read a brick's own points plus the matching regions of its
//     neighbours.
//   InsertPointsSubcell (V:4971-5092, P:109-118, P:218-315, P:677-694).
#include <algorithm>

#include "dev_common.cuh"

namespace gvdb2 {

namespace {

// gvdbInsertPoints (P:19-36): NOHIT positions and points outside every
// leaf get pnode = ID_UNDEFL; others take an atomic slot in their leaf.
__global__ void k_insert_points(PointsView pos, int64_t n, float3 trans, LeafLookup L, int32_t *pnode, int32_t *poff,
                                int32_t *gcnt) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 p = load_f3(pos, i);
    if (p.z == kNoHit) {
        pnode[i] = (int32_t)kUndefL;
        return;
    }
    int32_t leaf = leaf_at(L, p.x + trans.x, p.y + trans.y, p.z + trans.z);
    if (leaf < 0) {
        pnode[i] = (int32_t)kUndefL;
        return;
    }
    pnode[i] = leaf;
    poff[i] = atomicAdd(&gcnt[leaf], 1);
}

// gvdbSortPoints (P:59-72)
__global__ void k_sort_points(PointsView pos, int64_t n, float3 trans, const int32_t *pnode, const int32_t *poff,
                              int64_t nleaves, const uint32_t *goff, float *out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t nid = pnode[i];
    if (nid < 0 || nid >= nleaves) return;
    int64_t k = (int64_t)goff[nid] + poff[i];
    float3 p = load_f3(pos, i);
    out[3 * k + 0] = p.x + trans.x;
    out[3 * k + 1] = p.y + trans.y;
    out[3 * k + 2] = p.z + trans.z;
}

// Bins every point by the 8^3 cell that contains it and by its region in
// that cell: bin = cell * 27 + (rz * 3 + ry) * 3 + rx, cell = slot * m^3 +
// cell in the brick (-1 when no active brick contains it).  Per axis the
// region is 0 when the kernel's stencil reaches into the cell below (first
// tap < 0), 2 when it reaches into the cell above (last tap >= 8), else 1 (a
// stencil is narrower than a cell, so never both).  A cell's points so come
// ordered by region, and the points of a neighbour whose stencils reach a
// cell are a few contiguous runs of that neighbour's bin.  Bound by the latency
// of the leaf lookup and by an atomic add a point.  (One add for the points of a
// warp that share a bin: 16.7M lattice points 201 us against 176, 1M shell points
// 28 against 17, 16.7M points in random order 393 against 355.)
template <int KERNEL>
__device__ __forceinline__ int region_axis(float w, int cell_lo) {
    // first tap of Taps<KERNEL>::eval, relative to the cell's first voxel
    const int first = (int)floorf(w - 0.5f) - Taps<KERNEL>::LO - cell_lo;
    return first < 0 ? 0 : (first + Taps<KERNEL>::N - 1 >= kCell ? 2 : 1);
}

template <int KERNEL>
__global__ void k_bin_count(PointsView pos, int64_t n, float3 trans, LeafLookup L, const int32_t *leaf_slot, int m,
                            uint32_t *cnt, int32_t *pbin, int32_t *prank, uint32_t *cell_cnt) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kCntWords) cell_cnt[i] = 0; // for k_cell_list
    int32_t bin = -1;
    if (i < n) {
        float3 p = load_f3(pos, i);
        if (p.z != kNoHit) {
            const float w[3] = {p.x + trans.x, p.y + trans.y, p.z + trans.z};
            const int3 o = point_origin(pos, i);
            const int32_t leaf = leaf_at_o(L, w[0], w[1], w[2], o);
            const int32_t slot = leaf >= 0 ? leaf_slot[leaf] : -1;
            if (slot >= 0) {
                const int rm = (1 << L.g.log2r0) - 1; // local voxel = voxel mod res0
                const int vx = (int)w[0] + o.x, vy = (int)w[1] + o.y, vz = (int)w[2] + o.z;
                const int lx = vx & rm, ly = vy & rm, lz = vz & rm;
                // the cell's first voxel along each axis, in the point's grid coordinates
                const int rx = region_axis<KERNEL>(w[0], (vx & ~(kCell - 1)) - o.x);
                const int ry = region_axis<KERNEL>(w[1], (vy & ~(kCell - 1)) - o.y);
                const int rz = region_axis<KERNEL>(w[2], (vz & ~(kCell - 1)) - o.z);
                bin = (slot * m * m * m + cell_of_local(lx, ly, lz, m)) * kRegions + (rz * 3 + ry) * 3 + rx;
            }
        }
    }
    if (bin >= 0) {
        pbin[i] = bin;
        prank[i] = (int32_t)atomicAdd(cnt + bin, 1u);
    } else if (i < n) {
        pbin[i] = -1;
    }
}

// keys for the stable (deterministic) binning: bin id, unbinned last
__global__ void k_bin_keys(const int32_t *pbin, int64_t n, uint64_t *keys, int32_t *vals) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t b = pbin[i];
    keys[i] = b >= 0 ? (uint64_t)b : 0xFFFFFFFFull;
    vals[i] = (int32_t)i;
}

// Each binned point's entry of the bin order: perm[j] = i and, in the same
// pass, bin_pos[j] = its translated position and cloud index (as
// k_bin_pack_pos writes them; the positions are read in point order).
__global__ void k_bin_fill(const int32_t *pbin, const int32_t *prank, int64_t n, const uint32_t *off, int32_t *perm,
                           PointsView pos, float3 trans, float4 *bin_pos) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t b = pbin[i];
    if (b < 0) return;
    const int64_t j = (int64_t)off[b] + prank[i];
    perm[j] = (int32_t)i;
    const float3 q = load_f3(pos, i);
    const int32_t cloud = pos.cloud ? pos.cloud[i] : -1;
    bin_pos[j] = make_float4(q.x + trans.x, q.y + trans.y, q.z + trans.z, __int_as_float(cloud));
}

// bin_pos[j] = the translated position of the point at bin-order entry j
// (perm[j]) and its cloud index (-1 outside a batch), for the j below the
// number of binned points, reg_off[nreg].
__global__ void k_bin_pack_pos(const int32_t *perm, const uint32_t *reg_off, int64_t nreg, PointsView pos,
                               float3 trans, float4 *bin_pos) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= (int64_t)reg_off[nreg]) return;
    const int32_t p = perm[j];
    const float3 q = load_f3(pos, p);
    const int32_t cloud = pos.cloud ? pos.cloud[p] : -1;
    bin_pos[j] = make_float4(q.x + trans.x, q.y + trans.y, q.z + trans.z, __int_as_float(cloud));
}

// List the cells that hold points by class: heavy in `list`, light in `light`, huge
// as items (cell, slice) in `tiles`.
constexpr int64_t kCellCountReadback = 1 << 16; // cells

// Cells of at least `dense_min` points (dense_min > 0) are the scatter's dense
// cells: each gets a partial slot (part[c], -1 for the other cells), ceil(k / slice) work items (cell,
// slice, slices, accumulator slot) and, when that is more than one, an accumulator
// slot for its integer sums.  With rows_on the dense cells of kRowsMin to kRowsMax
// points are listed in `rows`, and their items apart in row_work.  cls gets each
// cell's class of sources (SrcEdges), blk[k * gridDim.x + b] how many of block b's
// cells are in class k, cnt[kCntSrc + k] how many of all.  Cells of at most `light` (<=
// kLightCell) points are light.  All of it depends on the cell, its brick and their
// neighbours alone, so that a cloud of a batch gets what a volume of its own gets;
// only the call's choice between rows and fixed point (default mode) counts cells
// of the whole batch.
// reg_off holds each (cell, region) bin's first entry; off[c] = reg_off[27 c], each
// cell's (c = ncell: the end), is written for the kernels that follow.
__global__ void k_cell_list(const uint32_t *reg_off, uint32_t *off, int64_t ncell, int32_t *list, int32_t *light, int2 *tiles,
                            int32_t *part, int32_t *rows, int4 *work, int4 *row_work, uint32_t *cnt, const int32_t *nbr27, int m,
                            uint32_t dense_min, uint32_t slice, uint32_t light_max, bool cubic, bool rows_on,
                            uint8_t *cls, SrcEdges E, uint32_t *blk) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t first = c <= ncell ? reg_off[c * kRegions] : 0u;
    if (c <= ncell) off[c] = first;
    const uint32_t k = c < ncell ? reg_off[(c + 1) * kRegions] - first : 0u;
    const int size = k == 0 ? -1 : (k > kHeavyCell ? kCntHuge : (k > light_max ? kCntHeavy : kCntLight));
    const unsigned act = __ballot_sync(0xffffffffu, size >= 0);
    if (size >= 0) {
        const uint32_t r = warp_agg_inc(cnt, (uint32_t)size, act);
        if (size == kCntLight) light[r] = (int32_t)c;
        else if (size == kCntHeavy) list[r] = (int32_t)c;
        else {
            const uint32_t ns = (k + kTilePts - 1) / kTilePts, t = atomicAdd(cnt + kCntTiles, ns);
            for (uint32_t i = 0; i < ns; i++) tiles[t + i] = make_int2((int32_t)c, (int32_t)i);
        }
    }
    const bool dense = dense_min > 0 && k >= dense_min;
    const unsigned dn = __ballot_sync(0xffffffffu, dense);
    int32_t slot = -1;
    if (dense) slot = (int32_t)warp_agg_inc(cnt, (uint32_t)kCntDense, dn);
    if (c < ncell) part[c] = slot;
    uint32_t reach = dense ? 0u : k;
    if (cubic && c < ncell) {
        int64_t slot;
        int cc[3];
        cell_coords(c, m, m * m * m, slot, cc[0], cc[1], cc[2]);
        uint32_t faces = 0;
#pragma unroll
        for (int f = 0; f < 6; f++) {
            int nc[3] = {cc[0], cc[1], cc[2]};
            const int a = f >> 1, d = (f & 1) * 2 - 1;
            nc[a] += d;
            int64_t ns = slot;
            if (nc[a] < 0 || nc[a] >= m) {
                const int step[3] = {1, 3, 9};
                ns = nbr27[slot * 27 + 13 + d * step[a]];
                nc[a] -= d * m;
            }
            if (ns < 0) continue;
            const int64_t n = ns * m * m * m + (nc[2] * m + nc[1]) * m + nc[0];
            const uint32_t kn = reg_off[(n + 1) * kRegions] - reg_off[n * kRegions];
            if (!(dense_min > 0 && kn >= dense_min)) faces += kn;
        }
        reach += (uint32_t)((uint64_t)faces * 3 / 16);
    }
    // one class a brick, by its cells' mean (of a block's cells, where it has more): the
    // cells of a brick share sectors of its rows, which two passes would write twice
    __shared__ uint32_t total[kListCells];
    const int unit = min(m * m * m, kListCells);
    total[threadIdx.x] = 0;
    __syncthreads();
    if (reach > 0) atomicAdd(&total[threadIdx.x / unit], min(reach, 1u << 20));
    __syncthreads();
    const uint32_t sum = total[threadIdx.x / unit];
    int mine = 0;
#pragma unroll
    for (int i = 0; i < kSrcClasses - 1; i++) mine += sum <= (uint32_t)(E.edge[i] * unit);
    if (mine == kSrcClasses - 1 && reach > (uint32_t)E.edge[0]) mine = 0; // too long for the last class
    if (c < ncell) cls[c] = (uint8_t)mine;
#pragma unroll
    for (int i = 0; i < kSrcClasses; i++) {
        const int n = __syncthreads_count(c < ncell && mine == i);
        if (threadIdx.x == 0) {
            blk[(int64_t)i * gridDim.x + blockIdx.x] = (uint32_t)n;
            if (n > 0) atomicAdd(cnt + kCntSrc + i, (uint32_t)n);
        }
    }
    const bool row = rows_on && dense && k >= (uint32_t)kRowsMin && k <= (uint32_t)kRowsMax;
    const unsigned rn = __ballot_sync(0xffffffffu, row);
    if (row) rows[warp_agg_inc(cnt, (uint32_t)kCntRows, rn)] = (int32_t)c;
    if (dense) {
        const uint32_t ns = (k + slice - 1) / slice;
        const uint32_t first = atomicAdd(cnt + (row ? kCntRowWork : kCntWork), ns);
        const int32_t acc = ns > 1 ? (int32_t)atomicAdd(cnt + kCntMulti, 1u) : -1;
        for (uint32_t i = 0; i < ns; i++)
            (row ? row_work : work)[first + i] = make_int4((int32_t)c, (int32_t)i, (int32_t)ns, acc);
    }
}

// The cells in the order that the owner-computes pass takes them: class by class, in
// cell order within a class.  Cells that run at a time so read the same neighbours'
// points, a block's warps have cells alike and the longest come first.  (In the order
// of atomics, by 256 or 1,024 cells, the cubic scatter takes 5 to 10% longer, in cell
// order with the classes mixed 1M shell points 93 us instead of 70.)  blk: per class
// and block of cells its cells or, `scanned`, how many come before them.
__global__ void __launch_bounds__(kListCells) k_owner_list(const uint8_t *cls, int64_t ncell, const uint32_t *blk,
                                                           bool scanned, int32_t *list) {
    __shared__ uint32_t count[kSrcClasses][kListCells / 32], sums[2][kSrcClasses][kListCells / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.x, nb = gridDim.x;
    const int64_t c = (int64_t)b * kListCells + threadIdx.x;
    const int mine = c < ncell ? cls[c] : -1;
    uint32_t before = 0; // within the warp
#pragma unroll
    for (int k = 0; k < kSrcClasses; k++) {
        const unsigned mask = __ballot_sync(0xffffffffu, mine == k);
        if (mine == k) before = __popc(mask & lanemask_lt());
        if (lane == 0) count[k][warp] = __popc(mask);
        if (scanned) continue;
        // at most kListCells blocks with cells
        const uint32_t n = (int)threadIdx.x < nb ? blk[k * nb + threadIdx.x] : 0u;
        const uint32_t s0 = __reduce_add_sync(0xffffffffu, (int)threadIdx.x < b ? n : 0u), s1 = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) sums[0][k][warp] = s0, sums[1][k][warp] = s1;
    }
    __syncthreads();
    uint32_t first = 0; // of the class
    for (int k = 0; k <= mine && !scanned; k++)
        for (int w = 0; w < kListCells / 32; w++) {
            if (k < mine) first += sums[1][k][w];
            if (k == mine) first += sums[0][k][w];
        }
    if (mine < 0) return;
    if (scanned) first = blk[(int64_t)mine * nb + b];
    for (int w = 0; w < warp; w++) before += count[mine][w];
    list[first + before] = (int32_t)c;
}

// The cells of class `first` and the later ones in cell order: k_scatter_light's list
// in volumes of many cells, where empty cells' writes and other cells' sums overlap.
// off: per class and block of cells how many come before them (k_owner_list).
__global__ void __launch_bounds__(kListCells) k_light_list(const uint8_t *cls, int64_t ncell, const uint32_t *off,
                                                           int first, int32_t *list) {
    __shared__ uint32_t count[kListCells / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.x, nb = gridDim.x;
    const int64_t c = (int64_t)b * kListCells + threadIdx.x;
    const bool in = c < ncell && cls[c] >= first;
    const unsigned mask = __ballot_sync(0xffffffffu, in);
    if (lane == 0) count[warp] = __popc(mask);
    __syncthreads();
    if (!in) return;
    uint32_t at = __popc(mask & lanemask_lt());
    for (int k = first; k < kSrcClasses; k++) at += off[(int64_t)k * nb + b] - off[(int64_t)k * nb];
    for (int w = 0; w < warp; w++) at += count[w];
    list[at] = (int32_t)c;
}

// gvdbSetFlagSubcell (P:109-118)
__global__ void k_sc_flag(const Node *leaves, int64_t n, uint32_t *flag) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flag[i] = leaves[i].mParent == kUndef64 ? 0u : 1u;
}

struct ScArgs {
    PointsView pos;
    int64_t n;
    float3 trans;
    float radius;
    int sc, scdim, scpb;
    int64_t num_sc;
    LeafLookup L;
    int64_t nleaves;
    const uint32_t *mapping; // a leaf's place among the listed ones (nullptr: its pool index)
    // pass 2 (InsertPointsSubcell_FP16): quantization ranges, velocities
    float3 pmin, prange, vmin, vrange;
    PointsView vel;
    uint16_t *q, *qvel;
};

// gvdbInsertSubcell_fp16's 16-bit quantization (P:195-203): (x - lo) /
// range * 65535 with the reference's approximate division, converted as a
// float-to-unsigned-short conversion does: toward zero, clamped, NaN to 0.
__device__ __forceinline__ uint16_t quantize16(float x, float lo, float range) {
    const float t = __fdividef(x - lo, range) * 65535.0f;
    if (!(t > 0.0f)) return 0; // also NaN
    return t >= 65535.0f ? (uint16_t)65535 : (uint16_t)t;
}

// gvdbCountSubcell (P:275-315, pass 0) / gvdbInsertSubcell (P:218-273,
// pass 1) / gvdbInsertSubcell_fp16 (P:154-216, pass 2).  The count pass
// tests the sign after adding trans, the insert pass before, the fp16 insert
// pass tests NOHIT and the sign on the translated position, all as in the
// reference; an insert never writes past the counted capacity of its
// subcell.  Bound by an atomic add a visit and, in the inserts, by the 12-byte
// entries they place.  The box's leaves are looked up once a brick, at most two
// an axis, and not once a subcell: 3M points at random, 64 a cell, 4^3 subcells and
// radius 2, 686 + 1,798 -> 329 + 1,574 us to count and insert; in cell order 498 + 624
// -> 266 + 512.  (Three subcells' adds along z before the first entry: 377 + 1,563 and
// 295 + 499, but 8^3 subcells 306 + 434 instead of 258 + 400.  Brick by brick, the
// lanes' loops diverge, and one add for the lanes of a warp that visit a subcell
// together was slower by half.)
template <int PASS>
__global__ void k_sc_visit(ScArgs A, uint32_t *cnt, const uint32_t *off, float *pnt) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    float3 p = load_f3(A.pos, i);
    float w[3];
    if (PASS == 2) {
        w[0] = p.x + A.trans.x;
        w[1] = p.y + A.trans.y;
        w[2] = p.z + A.trans.z;
        if (w[2] == kNoHit) return;
        if (w[0] < 0 || w[1] < 0 || w[2] < 0) return;
    } else if (p.z == kNoHit) {
        return;
    } else if (PASS == 0) {
        w[0] = p.x + A.trans.x;
        w[1] = p.y + A.trans.y;
        w[2] = p.z + A.trans.z;
        if (w[0] < 0 || w[1] < 0 || w[2] < 0) return;
    } else {
        if (p.x < 0 || p.y < 0 || p.z < 0) return;
        w[0] = p.x + A.trans.x;
        w[1] = p.y + A.trans.y;
        w[2] = p.z + A.trans.z;
    }
    int mn[3], mx[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        mn[a] = max(((int)(w[a] - A.radius) / A.sc) * A.sc, 0);
        // no brick lies past 2^30; a box there would step past the largest int
        mx[a] = (min((int)(w[a] + 1 + A.radius), 1 << 30) / A.sc) * A.sc;
        if (mx[a] < mn[a]) return;
    }
    const int lr = A.L.g.log2r0, rm = (1 << lr) - 1, ls = __ffs(A.sc) - 1; // a power of two, as it divides the brick
    // first subcell of a brick's subcells, or -1
    auto first_of = [&](int bx, int by, int bz) {
        const int32_t leaf = leaf_at_brick(A.L, bx, by, bz);
        if (leaf < 0 || leaf >= A.nleaves) return int64_t(-1);
        return (int64_t)(A.mapping ? A.mapping[leaf] : (uint32_t)leaf) * A.scpb;
    };
    auto place = [&](int64_t idx, uint32_t o) {
        const uint32_t first = off[idx];
        if (o >= off[idx + 1] - first) {
            atomicSub(&cnt[idx], 1u); // the list keeps its counted length
            return;
        }
        const int64_t at = (int64_t)first + o;
        if (PASS == 2) {
            A.q[3 * at + 0] = quantize16(w[0], A.pmin.x, A.prange.x);
            A.q[3 * at + 1] = quantize16(w[1], A.pmin.y, A.prange.y);
            A.q[3 * at + 2] = quantize16(w[2], A.pmin.z, A.prange.z);
            if (A.qvel) {
                const float3 u = load_f3(A.vel, i);
                A.qvel[3 * at + 0] = quantize16(u.x, A.vmin.x, A.vrange.x);
                A.qvel[3 * at + 1] = quantize16(u.y, A.vmin.y, A.vrange.y);
                A.qvel[3 * at + 2] = quantize16(u.z, A.vmin.z, A.vrange.z);
            }
        } else {
            pnt[3 * at + 0] = w[0];
            pnt[3 * at + 1] = w[1];
            pnt[3 * at + 2] = w[2];
        }
    };
    const int bx = mn[0] >> lr, by = mn[1] >> lr, bz = mn[2] >> lr;
    const int ex = (mx[0] >> lr) - bx, ey = (mx[1] >> lr) - by, ez = (mx[2] >> lr) - bz;
    if (ex > 1 || ey > 1 || ez > 1) { // a box over three bricks and more
        for (int sx = mn[0]; sx <= mx[0]; sx += A.sc)
            for (int sy = mn[1]; sy <= mx[1]; sy += A.sc)
                for (int sz = mn[2]; sz <= mx[2]; sz += A.sc) {
                    const int64_t f = first_of(sx >> lr, sy >> lr, sz >> lr);
                    const int64_t idx = f + ((((sz & rm) >> ls) * A.scdim + ((sy & rm) >> ls)) * A.scdim + ((sx & rm) >> ls));
                    if (f < 0 || idx >= A.num_sc) continue;
                    const uint32_t o = atomicAdd(&cnt[idx], 1u);
                    if (PASS != 0) place(idx, o);
                }
        return;
    }
    // the box's bricks, two an axis at most, each looked up once
    int64_t f[2][2][2];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int kx = k & 1, ky = (k >> 1) & 1, kz = k >> 2;
        f[kx][ky][kz] = kx <= ex && ky <= ey && kz <= ez ? first_of(bx + kx, by + ky, bz + kz) : int64_t(-1);
    }
    for (int sx = mn[0]; sx <= mx[0]; sx += A.sc) {
        const bool x1 = (sx >> lr) != bx;
        const int64_t g00 = x1 ? f[1][0][0] : f[0][0][0], g10 = x1 ? f[1][1][0] : f[0][1][0],
                      g01 = x1 ? f[1][0][1] : f[0][0][1], g11 = x1 ? f[1][1][1] : f[0][1][1];
        for (int sy = mn[1]; sy <= mx[1]; sy += A.sc) {
            const bool y1 = (sy >> lr) != by;
            const int64_t h0 = y1 ? g10 : g00, h1 = y1 ? g11 : g01;
            const int row = ((sy & rm) >> ls) * A.scdim + ((sx & rm) >> ls);
            for (int sz = mn[2]; sz <= mx[2]; sz += A.sc) {
                const int64_t h = (sz >> lr) != bz ? h1 : h0;
                const int64_t idx = h + ((sz & rm) >> ls) * (A.scdim * A.scdim) + row;
                if (h < 0 || idx >= A.num_sc) continue;
                const uint32_t o = atomicAdd(&cnt[idx], 1u);
                if (PASS != 0) place(idx, o);
            }
        }
    }
}

// gvdbCalcSubcellPos (P:677-694), a thread per subcell of every pool leaf
// (scpb subcells a leaf, 512 of them in a 32^3 brick).  Bound by its 16 bytes
// of stores a subcell; a thread per leaf that looped over its subcells left
// all but a few warps idle (150 bricks of 32^3: 313 us, 48 bricks: 177 us;
// a thread per subcell: 2 us).
__global__ void k_sc_pos(const Node *leaves, int64_t n, const uint32_t *mapping, int sc, int scdim, int scpb,
                         int64_t num_sc, int32_t *sc_nid, int32_t *sc_pos) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * scpb) return;
    const int64_t i = t / scpb;
    const int s = (int)(t - i * scpb);
    const Node &nd = leaves[i];
    if (nd.mParent == kUndef64) return;
    const int64_t idx = (mapping ? (int64_t)mapping[i] : i) * scpb + s;
    if (idx >= num_sc) return;
    sc_pos[3 * idx + 0] = nd.mPos[0] + s % scdim * sc;
    sc_pos[3 * idx + 1] = nd.mPos[1] + (s / scdim) % scdim * sc;
    sc_pos[3 * idx + 2] = nd.mPos[2] + (s / scdim / scdim) % scdim * sc;
    sc_nid[idx] = (int32_t)i;
}

} // namespace

gvdb2_status insert_points(Volume *v, int n, const float trans[3], int prefix) {
    if (v->pos.cloud) return fail(v, GVDB2_ERR_UNSUPPORTED, "batched clouds: the reference-mode point operations (InsertPoints, InsertPointsSubcell) take one cloud per volume");
    if (v->pool_cnt[0] == 0) return fail(v, GVDB2_ERR_STATE, "no topology");
    if (n < 0 || (n > 0 && (!v->pos.base || n > v->pos.count))) return fail(v, GVDB2_ERR_ARG, "bad point count");
    cudaStream_t s = v->stream;
    int64_t nl = v->pool_cnt[0];
    GV_CUDA(v, v->pnode.ensure(sizeof(int32_t) * (size_t)std::max(n, 1), s));
    GV_CUDA(v, v->poff.ensure(sizeof(int32_t) * (size_t)std::max(n, 1), s));
    GV_CUDA(v, v->gcnt.ensure(sizeof(int32_t) * (size_t)nl, s));
    GV_CUDA(v, cudaMemsetAsync(v->gcnt.p, 0, sizeof(int32_t) * (size_t)nl, s));
    GV_CUDA(v, cudaMemsetAsync(v->poff.p, 0, sizeof(int32_t) * (size_t)std::max(n, 1), s));
    float3 t = make_float3(trans[0], trans[1], trans[2]);
    LeafLookup L = make_lookup(v);
    if (n > 0)
        k_insert_points<<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(v->pos, n, t, L, v->pnode.as<int32_t>(),
                                                                    v->poff.as<int32_t>(), v->gcnt.as<int32_t>());
    GV_CUDA(v, cudaGetLastError());
    v->pnode_n = n;
    if (prefix) {
        GV_CUDA(v, v->goff.ensure(sizeof(uint32_t) * (size_t)(nl + 1), s));
        GV_TRY(exclusive_scan_u32(v, v->gcnt.as<uint32_t>(), v->goff.as<uint32_t>(), nl));
        GV_CUDA(v, v->psorted.ensure(sizeof(float) * 3 * (size_t)std::max(n, 1), s));
        if (n > 0)
            k_sort_points<<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(v->pos, n, t, v->pnode.as<int32_t>(),
                                                                      v->poff.as<int32_t>(), nl, v->goff.as<uint32_t>(),
                                                                      v->psorted.as<float>());
        GV_CUDA(v, cudaGetLastError());
    }
    return GVDB2_OK;
}

gvdb2_status light_list(Volume *v, int64_t ncell, int first) {
    const int g = grid_for(ncell + 1, kListCells, 1ll << 31);
    GV_CUDA(v, v->light_list.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(ncell, 1), v->stream));
    k_light_list<<<g, kListCells, 0, v->stream>>>(v->cell_cls.as<uint8_t>(), ncell,
                                                  v->cell_blk.as<uint32_t>() + (int64_t)kSrcClasses * g, first,
                                                  v->light_list.as<int32_t>());
    GV_CUDA(v, cudaGetLastError());
    return GVDB2_OK;
}

gvdb2_status bin_points(Volume *v, int kernel, int n, const float trans[3]) {
    Volume::BinKey &k = v->bin_key;
    // the regions depend on the kernel's stencil, so the bins do too
    if (k.valid && k.n == n && k.kernel == kernel && k.topo == v->topo_version && k.det == (v->deterministic != 0) &&
        k.pos.base == v->pos.base &&
        k.pos.stride == v->pos.stride && k.pos.offset == v->pos.offset && k.trans[0] == trans[0] &&
        k.trans[1] == trans[1] && k.trans[2] == trans[2] && k.tune[0] == v->tune_dense && k.tune[1] == v->tune_slice &&
        k.tune[2] == v->tune_light)
        return GVDB2_OK;
    if (!v->atlas_valid) return fail(v, GVDB2_ERR_STATE, "UpdateAtlas must follow the topology rebuild");
    if (n < 0 || (n > 0 && (!v->pos.base || n > v->pos.count))) return fail(v, GVDB2_ERR_ARG, "bad point count");
    cudaStream_t s = v->stream;
    const int m = v->res(0) / kCell; // cells per brick edge (bins are 8^3 cells)
    if (m < 1 || v->res(0) % kCell) return fail(v, GVDB2_ERR_UNSUPPORTED, "kernel splats need bricks of a multiple of 8 voxels");
    const int64_t nbins = v->atlas_last * m * m * m; // cells
    const int64_t nreg = nbins * kRegions;          // (cell, region) bins
    if (nreg >= INT32_MAX) return fail(v, GVDB2_ERR_CAPACITY, "more than 2^31 / 27 cells of 8^3 voxels");
    GV_CUDA(v, v->pbin.ensure(sizeof(int32_t) * (size_t)std::max(n, 1), s));
    GV_CUDA(v, v->prank.ensure(sizeof(int32_t) * (size_t)std::max(n, 1), s));
    GV_CUDA(v, v->perm.ensure(sizeof(int32_t) * (size_t)std::max(n, 1), s));
    GV_CUDA(v, v->bin_cnt.ensure(sizeof(uint32_t) * (size_t)(nreg + 1), s));
    GV_CUDA(v, v->reg_off.ensure(sizeof(uint32_t) * (size_t)(nreg + 1), s));
    GV_CUDA(v, v->bin_off.ensure(sizeof(uint32_t) * (size_t)(nbins + 1), s));
    GV_CUDA(v, cudaMemsetAsync(v->bin_cnt.p, 0, sizeof(uint32_t) * (size_t)(nreg + 1), s));
    GV_CUDA(v, v->cell_cnt.ensure(sizeof(uint32_t) * kCntWords, s));
    if (n == 0) GV_CUDA(v, cudaMemsetAsync(v->cell_cnt.p, 0, sizeof(uint32_t) * kCntWords, s));
    float3 t = make_float3(trans[0], trans[1], trans[2]);
    LeafLookup L = make_lookup(v);
    if (n > 0) {
        auto kc = kernel == GVDB2_KERNEL_TENT1 ? k_bin_count<GVDB2_KERNEL_TENT1> : k_bin_count<GVDB2_KERNEL_CUBIC2>;
        kc<<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(v->pos, n, t, L, v->leaf_slot.as<int32_t>(), m,
                                                     v->bin_cnt.as<uint32_t>(), v->pbin.as<int32_t>(),
                                                     v->prank.as<int32_t>(), v->cell_cnt.as<uint32_t>());
        GV_CUDA(v, cudaGetLastError());
    }
    GV_TRY(exclusive_scan_u32(v, v->bin_cnt.as<uint32_t>(), v->reg_off.as<uint32_t>(), nreg));
    if (n > 0 && v->deterministic) {
        // stable counting sort: a radix sort of (bin, point index) keeps each
        // bin's points in index order, independent of atomic timing; its key
        // buffer is the volume's scratch (grown like every other buffer)
        GV_CUDA(v, v->tmp_c.ensure(sizeof(uint64_t) * (size_t)n, s));
        uint64_t *keys = v->tmp_c.as<uint64_t>();
        k_bin_keys<<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(v->pbin.as<int32_t>(), n, keys, v->perm.as<int32_t>());
        GV_TRY(radix_sort_u64(v, keys, v->perm.as<int32_t>(), n, 0, 32));
    }
    // the points' positions in bin order: with the bin order itself from
    // the ranks, else from the sorted order
    GV_CUDA(v, v->bin_pos.ensure(sizeof(float4) * (size_t)std::max(n, 1), s));
    if (n > 0 && !v->deterministic) {
        k_bin_fill<<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(v->pbin.as<int32_t>(), v->prank.as<int32_t>(), n,
                                                               v->reg_off.as<uint32_t>(), v->perm.as<int32_t>(), v->pos,
                                                               t, v->bin_pos.as<float4>());
        GV_CUDA(v, cudaGetLastError());
    } else if (n > 0) {
        k_bin_pack_pos<<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(v->perm.as<int32_t>(), v->reg_off.as<uint32_t>(), nreg,
                                                                  v->pos, t, v->bin_pos.as<float4>());
        GV_CUDA(v, cudaGetLastError());
    }
    // the cells that hold points, by class (the gathers' grids), and the
    // scatter's dense cells with their work items
    GV_CUDA(v, v->cell_list.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(nbins, 1), s));
    GV_CUDA(v, v->cell_light.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(nbins, 1), s));
    // an item a huge cell, and one more for each kTilePts of its points
    GV_CUDA(v, v->cell_tiles.ensure(sizeof(int2) * (size_t)(n / (kHeavyCell + 1) + n / kTilePts + 1), s));
    GV_CUDA(v, v->cell_part.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(nbins, 1), s));
    GV_CUDA(v, v->cell_cls.ensure((size_t)std::max<int64_t>(nbins, 1), s));
    GV_CUDA(v, v->cell_owner.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(nbins, 1), s));
    // bounds from the point count: at most n / dense dense cells, and each
    // slice beyond a cell's first holds `slice` of its points
    const bool cubic = kernel == GVDB2_KERNEL_CUBIC2;
    // deterministic mode keeps the fixed-point sums, which no order changes
    const bool rows = cubic && !v->deterministic;
    const int64_t dmin = v->tune_dense, sl = v->tune_slice;
    v->dense_cap = dmin > 0 ? std::min<int64_t>(nbins, n / dmin) : 0;
    v->rows_cap = rows ? std::min<int64_t>(v->dense_cap, n / kRowsMin) : 0;
    v->rows_sorted = false;
    v->work_cap = dmin > 0 ? v->dense_cap + n / sl : 0;
    v->multi_cap = std::min<int64_t>(v->dense_cap, n / (sl + 1));
    GV_CUDA(v, v->rows_list.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(v->rows_cap, 1), s));
    GV_CUDA(v, v->row_work.ensure(sizeof(int4) * (size_t)std::max<int64_t>(v->rows_cap > 0 ? v->rows_cap + n / sl : 0, 1), s));
    GV_CUDA(v, v->part_work.ensure(sizeof(int4) * (size_t)std::max<int64_t>(v->work_cap, 1), s));
    v->heavy_grid = v->light_grid = 0;
    v->src_cells.fill(-1);
    v->cells_read = false;
    if (nbins == 0) GV_CUDA(v, cudaMemsetAsync(v->bin_off.p, 0, sizeof(uint32_t), s));
    if (nbins > 0) {
        const int g = grid_for(nbins + 1, kListCells, 1ll << 31);
        const bool few = nbins <= kCellCountReadback;
        GV_CUDA(v, v->cell_blk.ensure(sizeof(uint32_t) * (2 * kSrcClasses * (size_t)g + 1), s));
        k_cell_list<<<g, kListCells, 0, s>>>(v->reg_off.as<uint32_t>(), v->bin_off.as<uint32_t>(), nbins, v->cell_list.as<int32_t>(),
                                      v->cell_light.as<int32_t>(), v->cell_tiles.as<int2>(),
                                      v->cell_part.as<int32_t>(), v->rows_list.as<int32_t>(), v->part_work.as<int4>(), v->row_work.as<int4>(),
                                      v->cell_cnt.as<uint32_t>(),
                                      v->nbr27.as<int32_t>(), m, (uint32_t)dmin, (uint32_t)v->tune_slice, (uint32_t)v->tune_light,
                                      cubic, rows, v->cell_cls.as<uint8_t>(), few ? kSrcEdgesOne[cubic] : kSrcEdges[cubic],
                                      v->cell_blk.as<uint32_t>());
        GV_CUDA(v, cudaGetLastError());
        const uint32_t *blk = v->cell_blk.as<uint32_t>();
        if (!few) {
            uint32_t *off = v->cell_blk.as<uint32_t>() + (int64_t)kSrcClasses * g;
            GV_TRY(exclusive_scan_u32(v, blk, off, (int64_t)kSrcClasses * g));
            blk = off;
        }
        v->ordered = nbins > kOrderCells || n > kOrderPoints * nbins;
        if (v->ordered)
            k_owner_list<<<g, kListCells, 0, s>>>(v->cell_cls.as<uint8_t>(), nbins, blk, !few, v->cell_owner.as<int32_t>());
        GV_CUDA(v, cudaGetLastError());
        v->heavy_grid = nbins + n / kTilePts;
        v->light_grid = nbins;
        if (!few) {
            // many cells: size the grids by the cells of each class (one
            // small read) rather than by all cells
            uint32_t cw[kCntWords] = {0};
            GV_CUDA(v, cudaMemcpyAsync(cw, v->cell_cnt.p, sizeof(cw), cudaMemcpyDeviceToHost, s));
            GV_CUDA(v, cudaStreamSynchronize(s));
            v->heavy_grid = (int64_t)cw[kCntTiles] + cw[kCntHeavy];
            v->light_grid = cw[kCntLight];
            v->dense_cap = cw[kCntDense];
            v->rows_cap = cw[kCntRows];
            v->work_cap = (int64_t)cw[kCntWork] + cw[kCntRowWork];
            v->multi_cap = cw[kCntMulti];
            const bool sparse = 2 * (int64_t)cw[kCntSrc + kSrcClasses - 1] >= nbins;
            for (int i = 0; i < 4; i++) {
                v->src_classes[i] = sparse ? kOwnerClassesSparse : kOwnerClasses[cubic][i];
                v->src_cells[i] = 0;
                for (int k = 0; k < v->src_classes[i]; k++) v->src_cells[i] += cw[kCntSrc + k];
            }
        }
    }
    k.valid = true;
    k.det = v->deterministic != 0;
    k.kernel = kernel;
    k.n = n;
    k.topo = v->topo_version;
    k.pos = v->pos;
    for (int a = 0; a < 3; a++) k.trans[a] = trans[a];
    k.tune[0] = v->tune_dense;
    k.tune[1] = v->tune_slice;
    k.tune[2] = v->tune_light;
    return GVDB2_OK;
}

gvdb2_status insert_points_subcell(Volume *v, int sc, int n, float radius, const float trans[3], int *len,
                                   bool fp16) {
    if (v->pos.cloud) return fail(v, GVDB2_ERR_UNSUPPORTED, "batched clouds: the reference-mode point operations (InsertPoints, InsertPointsSubcell) take one cloud per volume");
    int res0 = v->res(0);
    if (sc <= 0 || res0 % sc) return fail(v, GVDB2_ERR_ARG, "subcell size must divide the brick resolution");
    if (n < 0 || (n > 0 && (!v->pos.base || n > v->pos.count))) return fail(v, GVDB2_ERR_ARG, "bad point count");
    int64_t num_brick = v->used_leaves;
    if (num_brick == 0) return fail(v, GVDB2_ERR_STATE, "InsertPointsSubcell yet no bricks exist");
    cudaStream_t s = v->stream;
    int scdim = res0 / sc, scpb = scdim * scdim * scdim;
    int64_t num_sc = (int64_t)scpb * num_brick, nmap = v->pool_cnt[0];
    v->sc_size = sc;
    v->sc_dim = scdim;
    v->sc_per_brick = scpb;
    v->num_sc = num_sc;
    GV_CUDA(v, v->sc_cnt.ensure(sizeof(uint32_t) * (size_t)(num_sc + 1), s));
    GV_CUDA(v, v->sc_off.ensure(sizeof(uint32_t) * (size_t)(num_sc + 1), s));
    GV_CUDA(v, v->sc_nid.ensure(sizeof(int32_t) * (size_t)num_sc, s));
    GV_CUDA(v, v->sc_pos.ensure(sizeof(int32_t) * 3 * (size_t)num_sc, s));
    // after a full rebuild every pool leaf is linked: its subcells lie at its pool
    // index, and every entry of the table is written
    const uint32_t *mapping = nullptr;
    if (!v->all_leaves_flagged) {
        GV_CUDA(v, v->sc_flag.ensure(sizeof(uint32_t) * (size_t)(nmap + 1), s));
        GV_CUDA(v, v->sc_map.ensure(sizeof(uint32_t) * (size_t)(nmap + 1), s));
        GV_CUDA(v, cudaMemsetAsync(v->sc_nid.p, 0, sizeof(int32_t) * (size_t)num_sc, s));
        GV_CUDA(v, cudaMemsetAsync(v->sc_pos.p, 0, sizeof(int32_t) * 3 * (size_t)num_sc, s));
        k_sc_flag<<<grid_for(nmap, 256, 1ll << 31), 256, 0, s>>>(v->pool_ptr(0), nmap, v->sc_flag.as<uint32_t>());
        GV_TRY(exclusive_scan_u32(v, v->sc_flag.as<uint32_t>(), v->sc_map.as<uint32_t>(), nmap));
        mapping = v->sc_map.as<uint32_t>();
    }
    uint32_t *cnt = v->sc_cnt.as<uint32_t>();
    GV_CUDA(v, cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (size_t)(num_sc + 1), s));
    ScArgs A;
    A.pos = v->pos;
    A.n = n;
    A.trans = make_float3(trans[0], trans[1], trans[2]);
    A.radius = radius;
    A.sc = sc;
    A.scdim = scdim;
    A.scpb = scpb;
    A.num_sc = num_sc;
    A.L = make_lookup(v);
    A.nleaves = nmap;
    A.mapping = mapping;
    A.pmin = make_float3(v->posmin[0], v->posmin[1], v->posmin[2]); // mPosMin, mPosRange (V:5452-5462)
    A.prange = make_float3(v->posmax[0] - v->posmin[0], v->posmax[1] - v->posmin[1], v->posmax[2] - v->posmin[2]);
    A.vmin = make_float3(v->velmin[0], v->velmin[1], v->velmin[2]);
    A.vrange = make_float3(v->velrange[0], v->velrange[1], v->velrange[2]);
    A.vel = v->vel;
    A.q = A.qvel = nullptr;
    v->sc_fp16 = fp16;
    v->sc_qvel_valid = false;
    if (n > 0) k_sc_visit<0><<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(A, cnt, nullptr, nullptr);
    GV_TRY(exclusive_scan_u32(v, cnt, v->sc_off.as<uint32_t>(), num_sc));
    uint32_t total = 0;
    GV_CUDA(v, cudaMemcpyAsync(&total, v->sc_off.as<uint32_t>() + num_sc, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    GV_CUDA(v, cudaStreamSynchronize(s));
    v->sc_len = total;
    if (len) *len = (int)total;
    if (total > 0) {
        GV_CUDA(v, cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (size_t)num_sc, s));
        if (fp16) {
            GV_CUDA(v, v->sc_q.ensure(sizeof(uint16_t) * 3 * (size_t)total, s));
            A.q = v->sc_q.as<uint16_t>();
            if (v->vel.base) { // velocities too, when SetPoints gave them (P:204-207)
                GV_CUDA(v, v->sc_qvel.ensure(sizeof(uint16_t) * 3 * (size_t)total, s));
                A.qvel = v->sc_qvel.as<uint16_t>();
                v->sc_qvel_valid = true;
            }
            if (n > 0)
                k_sc_visit<2><<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(A, cnt, v->sc_off.as<uint32_t>(), nullptr);
        } else {
            GV_CUDA(v, v->sc_pnt.ensure(sizeof(float) * 3 * (size_t)total, s));
            if (n > 0)
                k_sc_visit<1><<<grid_for(n, 256, 1ll << 31), 256, 0, s>>>(A, cnt, v->sc_off.as<uint32_t>(),
                                                                         v->sc_pnt.as<float>());
        }
    }
    k_sc_pos<<<grid_for(nmap * scpb, 256, 1ll << 31), 256, 0, s>>>(v->pool_ptr(0), nmap, mapping, sc,
                                                                   scdim, scpb, num_sc, v->sc_nid.as<int32_t>(),
                                                                   v->sc_pos.as<int32_t>());
    GV_CUDA(v, cudaGetLastError());
    return GVDB2_OK;
}

} // namespace gvdb2
