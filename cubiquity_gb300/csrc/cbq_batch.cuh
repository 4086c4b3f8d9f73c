// Job table of the multi-volume traversal kernel, shared by the batch API
// (cbq_batch.cu) and the request server (cbq_server.cu).
#pragma once

#include "cbq_flat.cuh"
#include "cbq_internal.hpp"

#include <cuda_runtime.h>

namespace cbq {
namespace dev {

// One job: a volume, its rays, its outputs and its query.  Jobs with rays are
// stored back to back in global ray index space starting at `first`.
struct JobDesc {
    const uint32_t* nodes;
    const float4* orig;
    const float4* dir;
    HitsOut out;
    uint64_t first;
    uint64_t count;
    QueryParams q;
    uint32_t occupied;  // bit k: SubDAG k is not empty
    const uint4* top;   // the volume's tables of upper cells
    SubDag sd[8];
};

}  // namespace dev

// Fills the parts of a JobDesc that come from the volume.
void fill_job_volume(dev::JobDesc& d, const cbq_dag* dag);

// Launch shape of the multi-volume kernel.
struct BatchLaunch {
    int block = 128;
    uint32_t refill = 16;            // idle lanes that trigger a warp's refill
    uint32_t steps = 8;              // walk iterations between a warp's checks for idle lanes
    bool shared_stack = true;        // descent stack in shared memory (stack_rows rows) instead of local
    int stack_rows = 0;              // max SubDAG height over the jobs
    const uint32_t* perm = nullptr;  // octant order (launch_batch_octant_sort), or null
    bool lod = true;                 // some job's query may stop at a footprint (max_footprint >= 0)
    bool spread = false;             // a small launch may be spread over the chip (spread_warp_rays)
    bool counter_zeroed = false;     // the work counter is already zero, in stream order
};

// Where the descent stack goes by default: in shared memory beside the jobs'
// prefix offsets while both fit the 48 KB that every block may have (a batch of
// 12 volumes: 264 us against 271 us with the local stack), else, for tables of
// thousands of jobs, in local memory.
inline bool batch_stack_in_shared(uint64_t njobs, int stack_rows, int block)
{
    return (njobs + 1) * 8 + (uint64_t)(stack_rows > 1 ? stack_rows : 1) * (uint64_t)block * 4 <= 48u * 1024u;
}

// Launches the persistent multi-volume kernel over `njobs` device-resident job
// descriptors holding `total` rays; all jobs' volumes have the compact layout,
// or none.  `counter` is zeroed on `stream` first, unless it is already.
cbq_status launch_batch_kernel(const dev::JobDesc* d_jobs, uint32_t njobs, uint64_t total, uint64_t* counter,
                               bool compact, int device, cudaStream_t stream, const BatchLaunch& bl);

// Groups each job's rays by octant (direction sign bits): perm[g] for g in a
// job's range [first, first + count) is a ray of the same job, all of its
// octant-0 rays first, then octant 1, and so on.  `scratch` holds 16 uint32
// per job (counts and cursors, zeroed here).
cbq_status launch_batch_octant_sort(const dev::JobDesc* d_jobs, uint32_t njobs, uint64_t total, uint32_t* scratch,
                                    uint32_t* perm, int device, cudaStream_t stream);

}  // namespace cbq
