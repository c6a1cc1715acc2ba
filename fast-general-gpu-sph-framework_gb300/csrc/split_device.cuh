// split_device.cuh — device code of the hybrid SMS/TRA split (rows A6-A8), run
// inside the grid sort's kernels (grid.cu): the performance model beside the
// pair scatter, the scan of its tile sums beside the small-cell sort, the
// compact index and the task descriptors after the big-cell sort.
//
// Reference behaviour (KemengHuang/Fast-General-GPU-SPH-framework):
//   performance model  src/io/gpu_model.cu:137-181
//                      (knCalculateBlockRequirementHybridMode)
//   TRA/SMS partition  src/grid/sph_arrangement.cu:87-107, 193-206, 358-384,
//                      1459-1482 (bucket = cell (TRA) or cell+numc (SMS);
//                      compact index = TRA particles, then SMS particles;
//                      "middle" = number of TRA particles)
//   task scan + tasks  src/grid/sph_arrangement.cu:1499-1500, 885-965
//                      (knArrangeSmsTasks)
//
// Design here: the work is indexed by OCCUPIED cells (compacted by the grid
// scan) instead of all numc cells, one scan of the triple {tasks, SMS
// particles, TRA particles} per occupied cell replaces the reference's second
// counting sort, and no host synchronisation is needed: counts stay on the
// device for the persistent density/force kernels.
#ifndef GSPH_SPLIT_DEVICE_CUH_
#define GSPH_SPLIT_DEVICE_CUH_

#include "gsph_internal.h"

namespace gsph {

namespace {

__device__ __forceinline__ int cell_n(const int32_t *start, int c) {
    return start[c + 1] - start[c];
}

// A6: SMS task count of one cell (gpu_model.cu:137-181, same neighbour
// bounds tests; the thresholds are the reference's unless tuned), with the
// cell's SMS and TRA particle counts: {req, sms, tra, 0}.
__device__ __forceinline__ int4 cell_model(int gidx, const int32_t *start,
                                           const SceneTable &T, int3 thr) {
    const SceneGeom G = geom_of_cell(T, gidx);
    const int idx = gidx - G.cbase;           // the scene's own cell index
    const int grid_x = G.gx, grid_y = G.gy;
    const int slice = grid_x * grid_y;
    const int numc = slice * G.gz;
    const int self = cell_n(start, gidx);
    int totaln = self;
    const int x = idx % grid_x;
    const int y = (idx / grid_x) % grid_y;
    if (x > 0) totaln += cell_n(start, gidx - 1);
    if (x + 1 < grid_x) totaln += cell_n(start, gidx + 1);
    if (y > 0) totaln += cell_n(start, gidx - grid_x);
    if (y + 1 < grid_y) totaln += cell_n(start, gidx + grid_x);
    if (idx >= slice) totaln += cell_n(start, gidx - slice);
    if (idx + slice < numc) totaln += cell_n(start, gidx + slice);
    int req;
    if (totaln < thr.x && self < thr.y)     // reference: 96, 15
        req = 0;
    else if (totaln < thr.z)                // reference: 60
        req = (self + 27) >> 5;
    else
        req = (self + 31) >> 5;
    const int sms = min(req * kSmsTaskParticles, self);
    return make_int4(req, sms, self - sms, 0);
}

__device__ __forceinline__ int4 add4(int4 a, int4 b) {
    return make_int4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ int4 shfl_up4(int4 v, int o) {
    return make_int4(__shfl_up_sync(0xFFFFFFFFu, v.x, o), __shfl_up_sync(0xFFFFFFFFu, v.y, o),
                     __shfl_up_sync(0xFFFFFFFFu, v.z, o), __shfl_up_sync(0xFFFFFFFFu, v.w, o));
}
__device__ __forceinline__ int4 shfl_down4(int4 v, int o) {
    return make_int4(__shfl_down_sync(0xFFFFFFFFu, v.x, o),
                     __shfl_down_sync(0xFFFFFFFFu, v.y, o),
                     __shfl_down_sync(0xFFFFFFFFu, v.z, o),
                     __shfl_down_sync(0xFFFFFFFFu, v.w, o));
}

// Exclusive scan, in place, of the int4 tile sums by one block; returns the
// grand total.
__device__ int4 scan_val_tiles(int4 *tiles, int ntiles) {
    __shared__ int4 ws[32];
    __shared__ int4 carry;
    if (threadIdx.x == 0) carry = make_int4(0, 0, 0, 0);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = int(blockDim.x >> 5);
    for (int base = 0; base < ntiles; base += blockDim.x) {
        const int t = base + threadIdx.x;
        const int4 v = t < ntiles ? tiles[t] : make_int4(0, 0, 0, 0);
        int4 x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int4 y = shfl_up4(x, o);
            if (lane >= o) x = add4(x, y);
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int4 w = lane < nw ? ws[lane] : make_int4(0, 0, 0, 0);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int4 y = shfl_up4(w, o);
                if (lane >= o) w = add4(w, y);
            }
            if (lane < nw) ws[lane] = w;
        }
        __syncthreads();
        const int4 wprefix = warp > 0 ? ws[warp - 1] : make_int4(0, 0, 0, 0);
        int4 excl = add4(carry, wprefix);
        excl = make_int4(excl.x + x.x - v.x, excl.y + x.y - v.y, excl.z + x.z - v.z, 0);
        if (t < ntiles) tiles[t] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = add4(excl, v);
        __syncthreads();
    }
    return carry;
}

// A6 + A7's scan inside a tile: the performance model of occupied cells
// [tile * kValTile, +kValTile) ({req, sms, tra} per cell), each cell's
// exclusive prefix inside the tile and the tile's sum; four consecutive cells
// per thread, kScanThreads threads.
__device__ __forceinline__ void model_tile(const Frame &f, const DevParams &P, int tile,
                                           int n) {
    __shared__ int4 ws[kScanThreads / 32];
    const int3 thr = make_int3(P.sparse_total, P.sparse_self, P.mid_total);
    const int first = tile * kValTile + threadIdx.x * kValItems;
    int4 v[kValItems];
    int4 s = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int q = 0; q < kValItems; ++q) {
        v[q] = first + q < n ? cell_model(f.occ_list[first + q], f.cell_start, f.scenes, thr)
                             : make_int4(0, 0, 0, 0);
        s = add4(s, v[q]);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int4 x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int4 y = shfl_up4(x, o);
        if (lane >= o) x = add4(x, y);
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    int4 run = make_int4(x.x - s.x, x.y - s.y, x.z - s.z, 0);
    for (int w = 0; w < warp; ++w) run = add4(run, ws[w]);
    bool any = false;
#pragma unroll
    for (int q = 0; q < kValItems; ++q) {
        if (first + q < n) {
            f.cell_val[first + q] = v[q];
            f.cell_prefix[first + q] = run;
        }
        any |= v[q].x > 0;
        run = add4(run, v[q]);
    }
    if (threadIdx.x == kScanThreads - 1) f.scan_tiles4[tile] = run;
    if (__syncthreads_or(any) && threadIdx.x == 0) atomicOr(&f.ctr->any_sms, 1);
}

// The scan of the tile sums by one block, which also sets the task count, the
// SMS particle count and the middle value. In a frame where no cell takes the
// SMS path there is nothing to compact: the grid scan has set the counts.
__device__ __forceinline__ void model_totals(const Frame &f) {
    if (!f.ctr->any_sms) return;
    const int4 total =
        scan_val_tiles(f.scan_tiles4, (f.ctr->num_occ + kValTile - 1) / kValTile);
    if (threadIdx.x == 0) {
        int tasks = total.x;
        if (tasks + 1 > f.task_capacity) {   // +1: odd-tail descriptor
            atomicOr(&f.ctr->err, kErrTaskCapacity);
            tasks = f.task_capacity - 1;
        }
        f.ctr->task_count = tasks;
        f.ctr->n_sms = total.y;
        f.ctr->middle = total.z;
    }
}

__host__ __device__ __forceinline__ uint16_t pack_bounds(int min_x, int max_x,
                                                         int min_y, int max_y,
                                                         int min_z, int max_z) {
    // packSmsTaskBounds, particle/particle_buffer.h:89-95
    return uint16_t(min_x | (max_x << 2) | (min_y << 4) | (max_y << 6) |
                    (min_z << 8) | (max_z << 10));
}

// {tasks, SMS particles, TRA particles} of the occupied cells before cell k.
__device__ __forceinline__ int4 cells_before(const Frame &f, int k) {
    return add4(f.scan_tiles4[k / kValTile], f.cell_prefix[k]);
}

// A8: the task descriptors of one occupied cell (particles [b, b + n), model
// values v, pre = cells_before), by `threads` threads numbered `t0`. micro(i)
// is the micro-cell part of the key of the cell's i-th sorted particle.
template <class Micro>
__device__ __forceinline__ void emit_tasks(const Frame &f, int cell, int b, int n, int4 v,
                                           int4 pre, int t0, int threads, Micro micro) {
    if (v.x == 0) return;
    const int task_count = f.ctr->task_count;
    const SceneGeom G = geom_of_cell(f.scenes, cell);
    const int local = cell - G.cbase;
    const uint16_t cx = uint16_t(local % G.gx);
    const uint16_t cy = uint16_t(local / G.gx % G.gy);
    const uint16_t cz = uint16_t(local / G.gx / G.gy);
    for (int t = t0; t < v.x; t += threads) {
        const int ti = pre.x + t;
        if (ti >= task_count) break;   // capacity guard (error already raised)
        const int off = t * kSmsTaskParticles;
        if (off >= kTaskOffsetLimit) {   // a cell beyond 2^24 particles
            atomicOr(&f.ctr->err, kErrTaskCapacity);
            break;
        }
        const uint32_t first_hash = micro(off);
        const uint32_t last_hash = micro(min(off + kSmsTaskParticles - 1, n - 1));
        const int min_x = (first_hash >> 4) & 3, max_x = (last_hash >> 4) & 3;
        const int min_z = (first_hash >> 2) & 3, max_z = (last_hash >> 2) & 3;
        const int min_y = first_hash & 3, max_y = last_hash & 3;
        gsph_block_task task;
        task.is_same = 0;
        task.cellid = cell;
        task.cell_pos[0] = cx;
        task.cell_pos[1] = cy;
        task.cell_pos[2] = cz;
        set_task_offset(task, off);
        task.cell_begin = b;
        task.cell_particle_count = n;
        task.xxi = int8_t(min_x);
        task.xxx = int8_t(max_x);
        if (min_x == max_x) {
            task.zzi = int8_t(min_z);
            task.zzz = int8_t(max_z);
            if (min_z == max_z) {
                task.yyi = int8_t(min_y);
                task.yyy = int8_t(max_y);
            } else {
                task.yyi = 0;
                task.yyy = 3;
            }
        } else {
            task.zzi = 0;
            task.zzz = 3;
            task.yyi = 0;
            task.yyy = 3;
        }
        task.paired_bounds =
            pack_bounds(task.xxi, task.xxx, task.yyi, task.yyy, task.zzi, task.zzz);
        f.tasks[ti] = task;
    }
}

// A7/A8: the compact index and the task descriptors of one occupied cell, by
// `threads` threads numbered `t0`.
template <class Micro>
__device__ __forceinline__ void emit_cell(const Frame &f, int cell, int b, int n, int4 v,
                                          int4 pre, int t0, int threads, Micro micro) {
    const int middle = f.ctr->middle;
    for (int j = t0; j < v.z; j += threads) f.compact[pre.z + j] = b + v.y + j;
    for (int j = t0; j < v.y; j += threads) f.compact[middle + pre.y + j] = b + j;
    emit_tasks(f, cell, b, n, v, pre, t0, threads, micro);
}

// The same for the small cells among 32 occupied cells from k0 on, by a warp:
// eight lanes write a cell's indices side by side (one thread per cell wrote
// to 32 sectors at a time: arrange of 3.94M particles with 8 SMS tasks 143.6 ->
// 140.9 us), a lane its cell's tasks. Tiles of the model without SMS cells, most
// of them where a sparse scene has grown a few, need no cell's values (133 us).
__device__ __forceinline__ void emit_small_cells(const Frame &f, int k0, int num_occ) {
    const int lane = threadIdx.x & 31;
    const int k = k0 + lane;
    const int tile = k0 / kValTile;
    const int before = f.scan_tiles4[tile].y;
    const int after = (tile + 1) * kValTile < num_occ ? f.scan_tiles4[tile + 1].y
                                                      : f.ctr->n_sms;
    int cell = 0, b = 0, n = 0;
    if (k < num_occ) {
        cell = f.occ_list[k];
        b = f.cell_start[cell];
        n = f.cell_start[cell + 1] - b;
    }
    if (before == after) {
        // no SMS cell in the tile: its particles follow one another in the
        // compact index, moved down by the SMS ones before them
        const int end = __shfl_sync(0xFFFFFFFFu, b + n, min(31, num_occ - 1 - k0));
        for (int i = __shfl_sync(0xFFFFFFFFu, b, 0) + lane; i < end; i += 32)
            f.compact[i - before] = i;
        return;
    }
    int4 v = make_int4(0, 0, 0, 0), pre = v;
    if (k < num_occ && n <= kSmallCellMax) {
        v = f.cell_val[k];
        pre = cells_before(f, k);
    }
    const int middle = f.ctr->middle;
#pragma unroll
    for (int q = 0; q < 32; q += 4) {
        const int src = q + (lane >> 3);
        const int sb = __shfl_sync(0xFFFFFFFFu, b, src);
        const int sms = __shfl_sync(0xFFFFFFFFu, v.y, src);
        const int tra = __shfl_sync(0xFFFFFFFFu, v.z, src);
        const int at = __shfl_sync(0xFFFFFFFFu, pre.z, src);
        for (int j = lane & 7; j < tra; j += 8) f.compact[at + j] = sb + sms + j;
        if (__any_sync(0xFFFFFFFFu, sms > 0)) {
            const int to = middle + __shfl_sync(0xFFFFFFFFu, pre.y, src);
            for (int j = lane & 7; j < sms; j += 8) f.compact[to + j] = sb + j;
        }
    }
    if (v.x > 0)
        emit_tasks(f, cell, b, n, v, pre, 0, 1, [&](int i) { return f.key[b + i]; });
}

}  // namespace

}  // namespace gsph

#endif  // GSPH_SPLIT_DEVICE_CUH_
