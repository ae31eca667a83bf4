// Internal launcher declarations shared by the kernel translation units and
// the C-ABI implementation (ensc_capi.cu).  Not installed; not part of the ABI.
#pragma once

#include "ensc_device.cuh"

#include <cuda_runtime.h>

#include <string>

namespace ensc {

// Launches a kernel of the cycle's sequence as programmatic dependent of the
// one before it in the stream: its blocks are set up while that one drains
// (cycle_kernel_enter).  Used up to the element pass: 1.2 us of a 36 us mixed
// cycle (262,144 elements), 2 of 135 us (48 instances).  The node passes are
// launched plainly: entering an SM that the element pass leaves, they would
// run beside its shared-memory carve-out, and the small L1 left by it holds
// fewer loads in flight (2,097,152 elements, mixed: 268 us a cycle against 232).
template <typename... P, typename... A>
inline void launch_cycle_kernel(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t st,
                                const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

constexpr int kElemThreads = 128;

// Minimum resident blocks per SM requested from the compiler for the element
// passes (register budget = 65536 / (128 * minb)); tuned on B200.
#ifndef ENSC_ELEM_MINB_FP64
#define ENSC_ELEM_MINB_FP64 3
#endif
#ifndef ENSC_ELEM_MINB_MIXED
#define ENSC_ELEM_MINB_MIXED 6
#endif
// the mixed element passes: warps per block, each with its own pipeline of
// 32-element tiles, and resident blocks per SM
#ifndef ENSC_MIXED_PIPE_WARPS
#define ENSC_MIXED_PIPE_WARPS 4
#endif
#ifndef ENSC_MIXED_PIPE_MINB
#define ENSC_MIXED_PIPE_MINB 4
#endif
// 1: the staged mixed element passes read A and the connectivity from the
// stage again for the force step instead of keeping them in registers
#ifndef ENSC_MIXED_REREAD
#define ENSC_MIXED_REREAD 1
#endif
#ifndef ENSC_NODE_BATCH_MINB_MIXED
#define ENSC_NODE_BATCH_MINB_MIXED 2
#endif
// the FP64 element passes: warps per block, each with its own pipeline of
// 32-element tiles, and resident blocks per SM
#ifndef ENSC_F64_PIPE_WARPS
#define ENSC_F64_PIPE_WARPS 4
#endif
#ifndef ENSC_F64_PIPE_MINB
#define ENSC_F64_PIPE_MINB 2
#endif
// 1: the FP64 element passes prefetch an element's second node records and vz
// into L1 once its connectivity is staged
#ifndef ENSC_F64_PREFETCH
#define ENSC_F64_PREFETCH 1
#endif
constexpr int kNodeThreads = 256;
constexpr int kCtlThreads = 256;

// ---- resident runs (ensc_run.cuh) ----
// Minima of one cycle's element phase, as ordered bits.
struct RunMins {
    unsigned long long dts, len;
};
// Grid-wide state of a resident run; between launches the minima are +inf and
// the rest zero.
struct alignas(128) RunSync {
    unsigned long long arrive;  // arrivals; 8 bits each from bit 48 and 56: blocks that saw an error in
                                // an element phase and in a node phase
    int32_t status, left;       // raised status bits, blocks that have left
    unsigned long long pad[14];
    RunMins mins[3];            // element phases of three cycles in turn
    unsigned long long pre;     // edge minimum of a cycle the total-time clamp may shorten
};
struct RunArgs {
    double step_end, pause;
    long long max_cycles;      // with arm: the limits of the step call (k_arm)
    int32_t arm;
    int32_t launch_cycles;     // most cycles of this launch
    int32_t tiles_per_warp;
};
// Launch geometry of an instance's resident runs; grid 0: the mesh does not
// fit, use the per-phase kernels.
struct RunPlan {
    int grid = 0, threads = 0, cluster = 0, tiles_per_warp = 0;
    int node_width = 1;        // nodes per thread of the node phase
    size_t smem = 0;
};
RunPlan plan_run_fp64(int64_t ne, int64_t nn, bool plastic, bool bt9, int sms);
RunPlan plan_run_mixed(int64_t ne, int64_t nn, bool plastic, int sms);
cudaError_t launch_run_fp64(const RunPlan& p, const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl,
                            const Partials& P, RunSync* sync, const RunArgs& a, cudaStream_t st);
cudaError_t launch_run_mixed(const RunPlan& p, const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl,
                             const Partials& P, RunSync* sync, const RunArgs& a, cudaStream_t st);

// FP64 (ensc_fp64.cu, built with -fmad=false)
void launch_element_fp64(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                         int grid, bool init, cudaStream_t st);
void launch_node_fp64(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                      int grid, cudaStream_t st);
int occupancy_element_fp64(bool plastic, bool bt9);
// nodes per thread of the node pass on the padded slot-major layout
#ifndef ENSC_NODE_GROUP_MIXED
#define ENSC_NODE_GROUP_MIXED 4
#endif
// resident blocks per SM requested for the node passes (register budget
// 65536 / (256 * minb)); tuned on B200
#ifndef ENSC_NODE_MINB_MIXED
#define ENSC_NODE_MINB_MIXED 2
#endif
#ifndef ENSC_NODE_MINB_FP64
#define ENSC_NODE_MINB_FP64 3
#endif
#ifndef ENSC_NODE_GROUP_FP64
#define ENSC_NODE_GROUP_FP64 1
#endif
constexpr int kNodeGroupFp64 = ENSC_NODE_GROUP_FP64;
constexpr int kNodeGroupMixed = ENSC_NODE_GROUP_MIXED;
// nodes per thread of the batched mixed node pass (with the nodes' rows
// loaded first, 4 spill there; 2 were 1% faster on the block as a batch and
// on a 64-instance sweep than 4 without loading first)
#ifndef ENSC_NODE_GROUP_BATCH_MIXED
#define ENSC_NODE_GROUP_BATCH_MIXED 2
#endif
constexpr int kNodeGroupBatchMixed = ENSC_NODE_GROUP_BATCH_MIXED;
int node_group_width(bool mixed_precision);
int occupancy_node_fp64();

// mixed precision (ensc_mixed.cu)
void launch_element_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                          int grid, bool init, cudaStream_t st, const PatchArrays& PA = PatchArrays{});
void launch_node_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                       int grid, cudaStream_t st, const PatchArrays& PA = PatchArrays{});
int occupancy_element_mixed(bool plastic, bool patch);
int occupancy_node_mixed();

// the last cycle's acceleration (compute_a), interleaved xyz per node, from
// the element forces the last force pass left in E.fe
void launch_acceleration_fp64(const ElemArrays& E, const NodeArrays& N, const Material& M, const Ctl* ctl,
                              double* a_aos, cudaStream_t st);
void launch_acceleration_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, const Ctl* ctl,
                               double* a_aos, cudaStream_t st, const PatchArrays& PA = PatchArrays{});

// batched instances (one launch per phase for all instances of a batch)
void launch_element_batch_fp64(const BatchTables& T, int grid, cudaStream_t st);
// threads per block of the batched node passes: kNodeThreads or half of it
void launch_node_batch_fp64(const BatchTables& T, int grid, int threads, cudaStream_t st);
int occupancy_element_batch_fp64(int tile_room);
int occupancy_node_batch_fp64(int threads);
void launch_element_batch_mixed(const BatchTables& T, int grid, bool patch, cudaStream_t st);
void launch_node_batch_mixed(const BatchTables& T, int grid, int threads, bool patch, cudaStream_t st);
int occupancy_element_batch_mixed(bool patch);
int occupancy_node_batch_mixed(int threads);
// elements and nodes per batch tile (element tiles are the tiles of 32, or
// patches; node tiles are one warp of node groups)
int batch_element_tile(bool patch);
int batch_node_tile(bool mixed_precision);
void launch_between_batch(const BatchTables& T, int slots, int mode, cudaStream_t st);
void launch_edge_prepass_batch(const BatchTables& T, int grid, cudaStream_t st);

// control (ensc_control.cu, built with -fmad=false)
// mode 0: begin the next cycle; 1: fold the energy partials; 2: fold them as the initial kinetic energy
void launch_between(Ctl* ctl, const Partials& P, int mode, cudaStream_t st);
void launch_edge_prepass(const ElemArrays& E, const NodeArrays& N, Ctl* ctl, int grid, cudaStream_t st);
// pause: the instance stops after the cycle in which its time reaches pause
// (dt is not clamped to it)
void launch_arm(Ctl* ctl, double step_end, long long max_cycles, cudaStream_t st, double pause = HUGE_VAL);
void launch_apply_bc_v(const NodeArrays& N, bool fp32_v, cudaStream_t st);
void launch_kinetic0(const NodeArrays& N, const Partials& P, Ctl* ctl, bool fp32_v, int grid, cudaStream_t st);
// Layout conversion between interleaved caller arrays and the device layout:
// node fields, reactions, and the element rows at `rows` of E.  `at` (may be null):
// entry e of the interleaved array is row position at[e] -- an element's stored
// position under the patch order.  A mixed instance's u rows hold x - u: its
// displacement is formed on the way out; on the way in the rows take u, between
// two calls of launch_reflect_rows (a <- x - a over the u rows).
enum class NodeField { X, U, V };
void launch_nodes_to_aos(const NodeArrays& N, NodeField field, bool mixed_precision, double* aos, cudaStream_t st);
void launch_aos_to_nodes(const double* aos, const NodeArrays& N, NodeField field, bool mixed_precision,
                         cudaStream_t st);
void launch_reactions_to_aos(const NodeArrays& N, double* aos, cudaStream_t st);
void launch_reflect_rows(const NodeArrays& N, cudaStream_t st);
void launch_elem_to_aos(const ElemArrays& E, const void* rows, int comps, bool src_fp32, double* aos, cudaStream_t st,
                        const int32_t* at = nullptr);
void launch_aos_to_elem(const double* aos, const ElemArrays& E, int comps, void* rows, bool dst_fp32, cudaStream_t st,
                        const int32_t* at = nullptr);

// thread-local message returned by ensc_last_error(NULL) (ensc_capi.cu)
void set_thread_error(const std::string& msg);

}  // namespace ensc
