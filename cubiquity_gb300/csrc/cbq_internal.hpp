// Internal declarations shared by the host (.cpp) and device (.cu) parts of
// libcbq.  Not part of the public ABI.
#pragma once

#include "../../include/cubiquity_gb300.h"
#include "cbq_counters.hpp"
#include "cbq_hostcopy.hpp"

#include <cstdint>
#include <memory>
#include <mutex>
#include <vector>

namespace cbq {

// Host-side findSubDAGs (raytracing.cpp:43-97).  Returns CBQ_ERR_BAD_DAG if a
// followed index is out of range.
cbq_status find_subdags(const uint32_t* nodes, uint64_t node_count, uint32_t root, cbq_subdag out[8]);

// Full structural check of a host node array.
cbq_status validate_nodes(const uint32_t* nodes, uint64_t node_count, uint32_t root);

// The largest t >= 0 with 1.0f / t > max_footprint (infinity for a negative
// max_footprint, -1 where there is none): for a child of size s, a power of
// two, and an exit distance t >= 0 in the range where the quotient neither
// overflows nor underflows, s / t > max_footprint exactly when t <= s * that.
float footprint_exit_max(float max_footprint);

// Device memory for a DAG: `whole` bytes (the node store, the walk's copy of it and the tables of
// upper cells), or, with a warning in the log, `store` bytes for the node store alone, where the
// walk takes the plain array (4 Mi bounce rays on terrain-4096 658 us instead of 526) and the
// batch kernel does not take the DAG (12 volumes 676 us instead of 213).  nullptr without memory
// for that either.
void* allocate_store(uint64_t whole, uint64_t store, void* (*allocate)(uint64_t bytes), bool* is_whole);

// printf-style message to the registered log handler (no-op without one).
void log(int level, const char* fmt, ...)
#if defined(__GNUC__)
    __attribute__((format(printf, 2, 3)))
#endif
    ;

// Checks that no internal node is reachable from a SubDAG root at height 0
// (which also excludes cycles), so a traversal never descends below the leaves.
cbq_status validate_heights(const uint32_t* nodes, uint64_t node_count, const cbq_subdag subdags[8]);

// Compact node store (CBQ_DAG_LAYOUT_COMPACT).  Every internal node reachable
// from a SubDAG root keeps only its occupied children, packed in slot order.  A
// reference to an internal node is (offset << 8) | occupancy mask, the offset
// counted in 8-byte units from the start of the store; unit 0 is unused, so
// every such reference is >= 256, above the material values, which children
// keep as they are.  A SubDAG rooted at a material m becomes a node with eight
// children m.  sd_ref[k] is SubDAG k's root reference (0 if empty).
// CBQ_ERR_CAPACITY when the store would exceed 2^24 units (128 MB).
cbq_status build_compact(const uint32_t* nodes, uint64_t node_count, const cbq_subdag subdags[8],
                         std::vector<uint32_t>& store, uint32_t sd_ref[8]);

// Resolves, on the current device, the device address of the fixed staging
// array of cbq_intersect_host_noalloc.  The lookup loads the module that holds
// the array, which is when the array takes its device memory; cbq_dag_create
// calls this so that the allocation happens there, never inside a
// cbq_intersect_host_noalloc call.
cbq_status noalloc_prepare(int device);

// Calls of cbq_intersect_host on one DAG that overlap in time (from several
// host threads) each take their own staging set, up to kHostStagesMax of them;
// beyond that they queue for one.
constexpr int kHostStagesMax = 4;

// Device staging and streams of one cbq_intersect_host call at a time: rays and
// hits, copied in and out in chunks on four streams (copy in, copy out, two for
// traversal) so that copies overlap the traversal.
struct HostStage {
    std::mutex lock;               // held by the call using this set
    void* d_stage = nullptr;
    uint64_t capacity = 0;         // rays
    struct CUstream_st* pipe[4] = {};  // cudaStream_t (this header is also compiled without CUDA)
    struct CUevent_st* pipe_ev[2 * kHostChunksMax] = {};  // cudaEvent_t
};

// The pathtracer's device memory, streams and events.  A DAG keeps one set between
// frames; a frame that finds it in use by another thread makes its own.  The memory
// kept is at most kPtKeptBytes over all DAGs of the process: a frame that would go
// beyond gives its own back when it is done.
constexpr uint64_t kPtKeptBytes = 1ull << 30;
// Waves that a frame is queued ahead of the last one whose ray count the host has looked at.
constexpr int kPtAhead = 4;
struct PtWorkspace {
    char* base = nullptr;
    uint64_t bytes = 0;
    uint64_t kept = 0;                     // its part of the memory kept by the process
    struct CUstream_st* wave = nullptr;    // extension waves and shading (higher priority)
    struct CUstream_st* shadow = nullptr;  // shadow waves
    struct CUevent_st* begin = nullptr;
    struct CUevent_st* shaded[kPtAhead] = {};  // a depth's shadow rays are written
    struct CUevent_st* traced[2] = {};     // ... and traced (their set may be written again)
    uint32_t* seen = nullptr;              // page-locked: the ray counts of the last kPtAhead waves shaded
};
void pt_workspace_release(PtWorkspace& w);

// Traversal of the rays that an earlier kernel on the stream counted at *n_dev (at
// most `most`), with a work counter that is zero in stream order.  Where
// takes_device_count(dag) is false the caller has to read the count itself.
bool takes_device_count(const cbq_dag* dag);
cbq_status intersect_device_count(const cbq_dag* dag, const cbq_rays* rays, uint64_t most, const uint32_t* n_dev,
                                  const cbq_query* query, const cbq_hits* hits, uint64_t* zeroed_counter,
                                  cbq_stream_t stream);

// Batch launches: 12 volumes, 2.2 M rays, shared stack: refill 16 at 8 iterations 264 us, refill 8
// 275 us.
constexpr uint32_t kBatchRefillDefault = 16;
constexpr int32_t kBatchStepsDefault = 8;

// Whether a configuration sets a launch shape of its own; otherwise small launches are spread
// over the chip (spread_warp_rays).  It depends on the values alone, so a configuration that was
// read and set again gives the same launches.
inline bool own_shape(const cbq_launch_config& c)
{
    return c.refill_min != 0 || c.steps != 0 || c.form != CBQ_FORM_PERSISTENT;
}
inline bool own_shape(const cbq_batch_config& c)
{
    return c.refill_min != kBatchRefillDefault || c.steps != kBatchStepsDefault || c.form != CBQ_FORM_PERSISTENT;
}

// The configurations that cbq_autotune times, as long as f(configuration) is true: every form,
// block size and stack; one thread per ray at four step counts, the refilled forms at the
// automatic shape and at three refills by four step counts.
template <typename F>
void for_each_tuned_config(const cbq_launch_config& base, F f)
{
    for (int form = CBQ_FORM_PLAIN; form <= CBQ_FORM_SORTED; form++)
        for (int block : {64, 128, 256})
            for (uint32_t refill : {0u, 8u, 16u, 24u}) {
                if (form == CBQ_FORM_PLAIN && refill != 0u) continue;  // refill unused
                for (int steps : {0, 4, 8, 16, 32})
                    for (int stack : {CBQ_STACK_SHARED, CBQ_STACK_LOCAL}) {
                        if ((steps == 0) != (refill == 0u && form != CBQ_FORM_PLAIN)) continue;
                        cbq_launch_config c = base;
                        c.kernel = CBQ_KERNEL_FLAT;
                        c.block = block;
                        c.refill_min = refill;
                        c.stack = stack;
                        c.form = form;
                        c.steps = steps;
                        c.registers = 0;
                        if (!f(c)) return;
                    }
            }
}

}  // namespace cbq

// The opaque DAG handle.
struct cbq_dag {
    uint32_t* d_nodes = nullptr;   // device: node_count * 8 words, or the compact store; in the same
                                   // allocation d_tagged and d_top
    uint32_t layout = CBQ_DAG_LAYOUT_REFERENCE;
    uint64_t device_bytes = 0;     // size of the device node store
    uint32_t sd_ref[8] = {};       // SubDAG roots as the device store refers to them
    // The store of the flat kernels' float form where d_nodes is the reference layout and has
    // fewer than 2^24 nodes: a copy of it whose references carry occupancy masks (made on the
    // device by cbq_dag_create; null where there is none), and the SubDAG roots in it.
    uint32_t* d_tagged = nullptr;
    uint32_t tagged_ref[8] = {};
    const uint32_t* walk_nodes() const { return d_tagged ? d_tagged : d_nodes; }
    uint32_t walk_root(int k) const { return d_tagged ? tagged_ref[k] : sd_ref[k]; }
    // Tables of the upper cells of SubDAGs of height 6 or more, in the walk's references
    // (dev::SubDag::top); null where there are none.
    uint32_t* d_top = nullptr;
    uint32_t top_index[8] = {};
    // The batch kernel takes tagged and compact stores; other DAGs are launched on their own.
    bool batch_ok() const { return flat_ok && (d_tagged || layout == CBQ_DAG_LAYOUT_COMPACT); }
    uint64_t node_count = 0;
    uint32_t root = 0;
    cbq_subdag subdags[8];
    int32_t max_height = 0;        // max SubDAG height (stack depth)
    int device = 0;
    bool flat_ok = false;          // float-position flat kernel applies (coordinates within +-2^21,
                                   // under 2^29 nodes); otherwise the integer-position form
    // Persistent refill, block 128, stack in shared memory; refill and steps 0: chosen by the
    // kernel from the rays (dev::WarpRefill).
    cbq_launch_config cfg{CBQ_KERNEL_AUTO, 0, 0, 0, CBQ_STACK_SHARED, CBQ_FORM_PERSISTENT, 0, 0};

    // Staging sets of cbq_intersect_host, created as concurrent calls need them.
    std::mutex stages_lock;
    std::vector<std::unique_ptr<cbq::HostStage>> stages;
    std::mutex pt_lock;  // held by the frame that uses `pt`
    cbq::PtWorkspace pt;
    cbq::CounterRings stream_counters;  // of cbq_intersect's persistent form
};
