// acfdtd_resident.cuh -- many steps per launch with the room's state held on chip (host interface).

#ifndef ACFDTD_RESIDENT_CUH
#define ACFDTD_RESIDENT_CUH

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "acfdtd_device.cuh"

namespace acf {

// How a room is cut into one brick per CTA: bx = planes * tx x planes by `rows` rows, all of z.
// A thread owns `planes` consecutive x planes of one (row, chunk) column.
struct ResidentPlan {
    int planes = 0;                // x planes per thread (0: the room does not fit)
    int tx = 0, rows = 0, chunks = 0, bx = 0, gx = 0, gy = 0;
    int threads = 0;               // per CTA, a multiple of 32
    int psi_shared = 0;            // relaxation states held in shared memory; the rest stay in HBM/L2
    size_t smem = 0, mailbox_bytes = 0;
};

// The plan for a room, or planes = 0 where no brick that holds it fits the device.
template <typename T>
ResidentPlan resident_plan(int nx, int ny, int nz, int n_relax, bool layer, int sms, size_t smem_limit);

template <typename T>
struct ResidentRun {
    Room<T> room;                  // the current copy, read before and written after the steps
    bool layer = false, walls = false;
    int n_relax = 0, steps = 0;
    void *mailbox = nullptr;       // plan.mailbox_bytes, zeroed when allocated
    int64_t *step_base = nullptr;  // device: absolute step of the first step
    uint32_t *epoch = nullptr;     // device, two words, zeroed when allocated
    uint64_t wait_limit_ns = kWaitLimitNs;
    int stop_step = -1;            // test hook: CTA 0 sends nothing from this step on
};

// Queue `run.steps` (>= 2) steps on `stream`: two launches.
template <typename T>
cudaError_t resident_launch(const ResidentPlan &plan, const ResidentRun<T> &run, int64_t first_step,
                            cudaStream_t stream);

}  // namespace acf

#endif
