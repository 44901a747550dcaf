// Internal to libcsmc: the device network handle behind csmc_net (shared by
// capi.cu and capi_batch.cu).
#pragma once
#include "../../include/csmc.h"
#include "include/csmc_net.h"
#include "kernels/sim.cuh"

#include <cuda_runtime.h>

#include <string>

// The geometry of one launch of the simulation kernels.
struct csmc_launch_plan {
    int family = 1;  // 0 = lane groups (lanes, comps_per_lane), 1 = one thread per run, 2 = one thread per run with
                     // the network read from global memory (the batch kernel with one job), 4 = class-coded
    int lanes = 0, comps_per_lane = 0, block = 256;
    size_t smem = 0;
    uint32_t state_stride = 0;
    bool state_in_global = false;
};

// A lane-group shape that fits the network, as launches choose among them.
struct csmc_group_shape {
    int lanes = 0, comps_per_lane = 0, block = 0;  // block: threads per CTA of a launch that fills the GPU
    uint32_t stride = 0;                           // shared memory of one group's run state
    int warps = 0;                                 // resident warps per SM at that block
};

struct csmc_net {
    int device = 0;
    uint8_t *d_blob = nullptr;
    uint32_t bytes = 0;       // staged bytes (multiple of 16)
    csmc_net_header h{};
    uint32_t clock_base = csmc::kNoClockBase;  // the clocks are consecutive variables from this one on
    unsigned long long *d_scratch = nullptr;
    // internal per-run buffers used when the caller passes none
    uint8_t *d_flags = nullptr;
    double *d_values = nullptr;
    uint64_t cap_runs = 0;
    double *d_partials = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    csmc_launch_plan plan;     // the plan set by csmc_set_plan, else the default of launches that fill the GPU
    bool plan_forced = false;  // csmc_set_plan: every launch uses `plan`
    csmc_launch_plan own_plan;  // the default `plan` had before csmc_set_plan
    csmc_group_shape shapes[6];  // lane-group shapes for launches that do not fill the GPU one thread per run
    int n_shapes = 0;
    int sms = 0;               // SMs of the device
    int thread_warps = 0;      // resident warps per SM of the default plan when it runs one thread per run (0: it does not)
    bool slots = false;
    bool loc8 = false;     // every automaton has at most 256 locations
    bool classes = false;  // delay descriptors carry race classes
    bool all_classed = false;  // every location belongs to a race class
    uint32_t class_src[CSMC_RACE_CLASSES] = {};  // 1/rate source of each class (SimParams::class_src)
    uint8_t *d_state = nullptr;  // thread-per-run state slabs (global-state plans)
    size_t state_bytes = 0;
    csmc::BatchJob *d_job = nullptr;  // family 2: the one-job table
    // importance sampling
    bool is_plain = false;  // every location is exponential (a literal or a rate program) or zero-delay
    csmc::MlpParams *d_mlp = nullptr;  // the proposal network
    double *d_wvals = nullptr;         // per run: flag * likelihood ratio
    uint8_t *d_is_flags = nullptr;
    uint64_t is_cap = 0;
    bool is_tc = false;  // importance sampling: theta by warp-level MMAs (false: the oracle-identical CUDA-core evaluation)
    bool is_feat_set = false;   // importance sampling: a feature source was chosen (else the default)
    csmc::MlpFeatures is_feat{};
    // importance sampling one thread per run (sim_is_coded.cuh): the tilt
    // groups of the network (is_groups < 0: the network does not qualify)
    int is_groups = -1;
    bool is_all_grouped = false;  // every location in a tilt group
    uint64_t is_group_map = 0;
    uint32_t is_group_l = 0;
    uint32_t is_group_src[CSMC_IS_GROUPS] = {};
    int is_kernel = 0;  // 0: thread per run where the network qualifies, 3: always one warp per run
    uint32_t *d_theta_cache = nullptr;  // thread-per-run kernel: the device-wide theta cache
    uint32_t theta_gen = 0;             // generation of the cached parameter block (0: none yet)
    unsigned char theta_params[CSMC_MLP_PARAM_BYTES] = {};  // the parameter block of that generation
};

namespace csmc {
inline NetLayout layout_of(const csmc_net &n) {
    NetLayout l = layout_of(n.h);
    l.clock_base = n.clock_base;
    return l;
}
void set_last_error(const std::string &m);  // capi.cu
}
