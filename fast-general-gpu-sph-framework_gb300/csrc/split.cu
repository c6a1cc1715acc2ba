// split.cu — the pairing of the SMS tasks (row A9). The performance model, the
// TRA/SMS partition and the task descriptors (A6-A8) are in split_device.cuh.
//
// Reference behaviour (KemengHuang/Fast-General-GPU-SPH-framework):
//   pairing            src/grid/sph_arrangement.cu:966-1022 (judgeTask)
#include <algorithm>

#include "split_device.cuh"

namespace gsph {

namespace {

// One pair (first, first + 1) of the historical same-cell pairing.
__device__ __forceinline__ void judge_pair(gsph_block_task *__restrict__ tasks,
                                           int first, int task_count) {
    const int second = first + 1;
    gsph_block_task a = tasks[first];
    if (second >= task_count) {
        // Odd tail (sph_arrangement.cu:976-991): a fabricated descriptor of
        // the next 32 particles of the same cell. Fields the reference leaves
        // stale are copied from the last task here.
        gsph_block_task t = a;
        a.is_same = 1;
        t.is_same = 1;
        set_task_offset(t, task_offset(a) + kSmsTaskParticles);
        tasks[first] = a;
        tasks[second] = t;
        return;
    }
    gsph_block_task b = tasks[second];
    if (a.cellid != b.cellid) {
        tasks[first].is_same = 0;
        tasks[second].is_same = 0;
        return;
    }
    int pmin_z = a.zzi, pmax_z = a.zzz;
    if (a.xxi == b.xxx) {
        pmax_z = b.zzz;
    } else {
        pmin_z = 0;
        pmax_z = 3;
    }
    tasks[first].is_same = 1;
    tasks[second].is_same = 1;
    tasks[first].paired_bounds =
        pack_bounds(a.xxi, b.xxx, a.yyi, a.yyy, pmin_z, pmax_z);
}

// A9: historical same-cell pairing of tasks (2k, 2k+1), odd-tail descriptor.
__global__ void __launch_bounds__(128)
k_judge(gsph_block_task *__restrict__ tasks, const Counters *ctr) {
    const int task_count = ctr->task_count;
    for (int pair = blockIdx.x * blockDim.x + threadIdx.x; (pair << 1) < task_count;
         pair += gridDim.x * blockDim.x)
        judge_pair(tasks, pair << 1, task_count);
}

}  // namespace

void launch_judge(const Frame &f, int max_occ, int num_sms, cudaStream_t s) {
    if (f.n <= 0 || max_occ <= 0) return;   // no tasks made
    const int max_pairs = (f.task_capacity + 1) / 2;
    k_judge<<<std::min((max_pairs + 127) / 128, num_sms * 8), 128, 0, s>>>(f.tasks,
                                                                          f.ctr);
}

}  // namespace gsph
