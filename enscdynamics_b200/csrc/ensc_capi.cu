// C ABI of the GPU stepper (include/ensc_gpu.h).
//
// Host-side responsibilities, in reference terms:
//   ensc_create   exDyna3D::init() (Explicit3D/source/exDyna3D.cpp:105-142):
//                 element constants and lumped mass (compute_invMassMatrix,
//                 :492-515), the node-to-element gather tables that replace the
//                 8 slot vectors of add_inForce_to_rhs (:523-639), device
//                 allocation, and the init force pass with dt = 0 that seeds
//                 the stable time step.
//   ensc_set_bcs  setCurrentStep's boundary update (:1760-1940, :1911).
//   ensc_step     run()'s loop body (:86-100): resident runs where the mesh fits on
//                 chip, else CUDA graphs of cycles and up to half a graph's
//                 cycles one by one.
//   ensc_download copies state back in the reference's array layouts.
#include "ensc_gpu.h"
#include "ensc_device.cuh"
#include "ensc_kernels.h"
#include "ensc_instance.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

using ensc::Ctl;

struct ensc_handle {
    int device = 0;
    int precision = ENSC_FP64;
    bool plastic = false;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    cudaStream_t cap_stream = nullptr;
    int64_t nn = 0, ne = 0, nn_pad = 0;
    void* arena = nullptr;
    size_t arena_bytes = 0;
    double* staging = nullptr;     // device AoS staging for up/download
    bool staging_owned = false;
    size_t staging_bytes = 0;
    ensc::ElemArrays E{};
    ensc::NodeArrays N{};
    ensc::PatchArrays PA{};        // patch assembly tables (null: slot assembly)
    ensc::Material M{};
    ensc::Partials P{};
    Ctl* ctl = nullptr;            // device
    Ctl* ctl_host = nullptr;       // pinned mirror
    int grid_e = 1, grid_n = 1;
    int chunk = 32;
    cudaGraphExec_t graph = nullptr;   // cycles of the per-phase kernels
    ensc::RunPlan run{};               // resident runs (grid 0: the graph)
    ensc::RunSync* sync = nullptr;
    bool kinetic0_done = false;
    double* amp = nullptr;         // device gravity amplitude table
    // output snapshots (ensc_snapshot_begin / ensc_snapshot_wait): a device
    // buffer of AoS fields and the control block, copied on copy_stream into
    // two pinned host buffers used in turn
    double* snap_dev = nullptr;
    size_t snap_bytes = 0;
    double* snap_host[2] = {nullptr, nullptr};
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t snap_captured = nullptr;
    cudaEvent_t snap_landed[2] = {nullptr, nullptr};
    int64_t snap_count = 0;
    bool fe_valid = false;         // fe holds the last force pass's element forces
    int64_t n_patches = 0, n_partials = 0;  // patch assembly
    std::string err;
};

namespace {

thread_local std::string g_create_error;

struct DevGuard {
    int prev = -1;
    explicit DevGuard(int d) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != d) cudaSetDevice(d);
    }
    ~DevGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

int set_err(ensc_handle* h, int code, const std::string& msg) {
    if (h) h->err = msg;
    else g_create_error = msg;
    return code;
}

int cuda_err(ensc_handle* h, const char* what, cudaError_t e) {
    std::string m = std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    return set_err(h, e == cudaErrorMemoryAllocation ? ENSC_ERR_OOM : ENSC_ERR_CUDA, m);
}

#define CK(h, call)                                   \
    do {                                              \
        cudaError_t _e = (call);                      \
        if (_e != cudaSuccess) return cuda_err((h), #call, _e); \
    } while (0)


// Copies a host vector to the device on the handle's stream, so that the
// kernels launched there after it see the data: a plain cudaMemcpy from
// pageable memory may return before its DMA lands, and it is not ordered
// with the handle's non-blocking stream.  (A pageable source is staged
// before the call returns, so the vector may go away after it.)
template <typename T>
int upload(ensc_handle* h, void* dst, const std::vector<T>& src) {
    if (src.empty()) return ENSC_OK;
    CK(h, cudaMemcpyAsync(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
    return ENSC_OK;
}

bool mixed(const ensc_handle* h) { return h->precision == ENSC_MIXED; }

void launch_element(ensc_handle* h, bool init, cudaStream_t st) {
    if (mixed(h)) ensc::launch_element_mixed(h->E, h->N, h->M, h->ctl, h->P, h->grid_e, init, st, h->PA);
    else ensc::launch_element_fp64(h->E, h->N, h->M, h->ctl, h->P, h->grid_e, init, st);
}

void launch_node(ensc_handle* h, cudaStream_t st) {
    if (mixed(h)) ensc::launch_node_mixed(h->E, h->N, h->M, h->ctl, h->P, h->grid_n, st, h->PA);
    else ensc::launch_node_fp64(h->E, h->N, h->M, h->ctl, h->P, h->grid_n, st);
}

// The per-phase kernels of one cycle.
void launch_cycle(ensc_handle* h, cudaStream_t st) {
    ensc::launch_between(h->ctl, h->P, 0, st);
    ensc::launch_edge_prepass(h->E, h->N, h->ctl, h->grid_e, st);
    launch_element(h, false, st);
    launch_node(h, st);
}

int build_graph(ensc_handle* h) {
    if (h->graph) {
        cudaGraphExecDestroy(h->graph);
        h->graph = nullptr;
    }
    cudaGraph_t g = nullptr;
    CK(h, cudaStreamBeginCapture(h->cap_stream, cudaStreamCaptureModeThreadLocal));
    for (int c = 0; c < h->chunk; ++c) launch_cycle(h, h->cap_stream);
    cudaError_t e = cudaStreamEndCapture(h->cap_stream, &g);
    if (e != cudaSuccess) return cuda_err(h, "cudaStreamEndCapture", e);
    e = cudaGraphInstantiate(&h->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_err(h, "cudaGraphInstantiate", e);
    return ENSC_OK;
}

// Most cycles of one resident-run launch (tens of ms on the meshes that run
// resident): the host looks at the control block between launches.
constexpr int64_t kRunCycles = 4096;

// Before kernels that fill the partial slots in another way than the cycles
// before them: folds what those left, and leaves no kinetic energy in slots that
// the kernels to come may not fill (a resident run fills one per block of its
// grid, the node pass and the initial sum grid_n of them).
int settle_energy(ensc_handle* h) {
    ensc::launch_between(h->ctl, h->P, 1, h->stream);
    CK(h, cudaGetLastError());
    CK(h, cudaMemsetAsync(h->P.node, 0, h->P.n_node_blocks * sizeof(double), h->stream));
    return ENSC_OK;
}

// The launches that rebuild what a handle steps with after its material or
// loads changed: the graph carries them by value, a resident run takes them
// with every launch.
int loads_changed(ensc_handle* h) { return h->graph ? build_graph(h) : ENSC_OK; }

// Enqueues up to `cycles` cycles of a step call: its first (arm, which sets
// the call's limits: max_cycles in all) or a later part.
int enqueue_cycles(ensc_handle* h, int64_t cycles, bool arm, int64_t max_cycles, double step_end, double pause) {
    // in a stream under capture every launch form refuses, not the graph's alone:
    // the cycles would be recorded with this call's limits, and none would run
    cudaStreamCaptureStatus capture;
    CK(h, cudaStreamIsCapturing(h->stream, &capture));
    if (capture != cudaStreamCaptureStatusNone)
        return cuda_err(h, "step call", cudaErrorStreamCaptureUnsupported);
    if (h->run.grid) {
        int64_t left = cycles;
        while (left > 0) {
            const int64_t n = std::min(left, kRunCycles);
            ensc::RunArgs a{step_end, pause, max_cycles, arm ? 1 : 0, static_cast<int32_t>(n), h->run.tiles_per_warp};
            const cudaError_t e =
                mixed(h) ? ensc::launch_run_mixed(h->run, h->E, h->N, h->M, h->ctl, h->P, h->sync, a, h->stream)
                         : ensc::launch_run_fp64(h->run, h->E, h->N, h->M, h->ctl, h->P, h->sync, a, h->stream);
            if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources) {
                // fewer SMs are open to this process than the device has:
                // the per-phase kernels need no resident grid
                cudaGetLastError();
                h->run = ensc::RunPlan{};
                if (int rs = settle_energy(h)) return rs;
                break;
            }
            if (e != cudaSuccess) return cuda_err(h, "resident run", e);
            arm = false;
            left -= n;
        }
        h->fe_valid = true;
        if (left == 0) return ENSC_OK;
        cycles = left;
    }
    // Whole graphs, then up to half a graph's cycles one by one: past the call's
    // last cycle a graph's kernels still take about 8 us a cycle to find nothing
    // to do, and their launches about as much host time (a call of one cycle,
    // 262,144 elements mixed: 221 us as a graph, 62 by itself; of 16: 648 and 611).
    int64_t graphs = cycles / h->chunk, single = cycles % h->chunk;
    if (2 * single > h->chunk) {
        graphs += 1;
        single = 0;
    }
    if (graphs && !h->graph)
        if (int rc = build_graph(h)) return rc;
    if (arm) ensc::launch_arm(h->ctl, step_end, max_cycles, h->stream, pause);
    for (int64_t i = 0; i < graphs; ++i) CK(h, cudaGraphLaunch(h->graph, h->stream));
    for (int64_t i = 0; i < single; ++i) launch_cycle(h, h->stream);
    CK(h, cudaGetLastError());
    h->fe_valid = true;
    return ENSC_OK;
}

int read_ctl(ensc_handle* h) {
    CK(h, cudaMemcpyAsync(h->ctl_host, h->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    return ENSC_OK;
}

int status_code(ensc_handle* h, int32_t st) {
    if (st & ensc::ST_NONFINITE) return set_err(h, ENSC_ERR_NONFINITE, "non-finite nodal state detected");
    if (st & ensc::ST_INVERTED) return set_err(h, ENSC_ERR_INVERTED, "element with J <= 0 detected");
    if (st & ensc::ST_BAD_DT) return set_err(h, ENSC_ERR_NONFINITE, "stable time step is not positive");
    if (st & ensc::ST_TIMEOUT) return set_err(h, ENSC_ERR_TIMEOUT, "a bounded wait for staged element data expired");
    return ENSC_OK;
}

void fill_report(const ensc_handle* h, int64_t before, ensc_step_report* r) {
    if (!r) return;
    const Ctl& c = *h->ctl_host;
    r->time = c.time;
    r->dt_i = c.dt_i;
    r->dt_i_1 = c.dt_i_1;
    r->cycles = c.cycles_done - before;
    r->total_cycles = c.cycles_done;
    r->status = (c.status & ensc::ST_TIMEOUT) ? ENSC_ERR_TIMEOUT
                : (c.status & ensc::ST_INVERTED) ? ENSC_ERR_INVERTED
                : c.status ? ENSC_ERR_NONFINITE : ENSC_OK;
    r->done = c.time < c.step_end ? 0 : 1;
    std::memcpy(&r->dt_stable_min, &c.dts_next, sizeof(double));
}

}  // namespace

namespace ensc {
void set_thread_error(const std::string& msg) { g_create_error = msg; }
}  // namespace ensc

extern "C" {

int ensc_abi_version(void) { return ENSC_ABI_VERSION; }

const char* ensc_last_error(const ensc_handle* h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int ensc_create(const ensc_mesh_desc* mesh, const ensc_material* mat, const ensc_params* params,
                ensc_handle** out) {
    if (!out) return set_err(nullptr, ENSC_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (!mesh || !mat || !params) return set_err(nullptr, ENSC_ERR_ARG, "mesh, material and params are required");
    if (params->precision != ENSC_FP64 && params->precision != ENSC_MIXED)
        return set_err(nullptr, ENSC_ERR_ARG, "unsupported precision");
    if (!(params->factor_timestep > 0.0)) return set_err(nullptr, ENSC_ERR_ARG, "factor_timestep must be > 0");
    const bool mx = params->precision == ENSC_MIXED;
    ensc::InstanceHost ih;
    std::string perr;
    int rc = ensc::instance_prepare(mesh, mat, mx, params->assembly, ih, perr);
    if (rc) return set_err(nullptr, rc, perr);
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= params->device || params->device < 0)
        return set_err(nullptr, ENSC_ERR_NODEVICE, "no usable CUDA device");

    ensc_handle* h = new ensc_handle();
    h->device = params->device;
    h->precision = params->precision;
    h->plastic = ih.plastic;
    h->nn = ih.nn;
    h->ne = ih.ne;
    h->nn_pad = ih.nn_pad;
    h->chunk = params->graph_chunk > 0 ? params->graph_chunk : 32;
    DevGuard dg(h->device);
    auto fail = [&](int code) {
        g_create_error = h->err;
        ensc_destroy(h);
        return code;
    };

    // ---- launch geometry: persistent grids of (resident blocks per SM) x SMs ----
    cudaDeviceProp prop{};
    if (cudaGetDeviceProperties(&prop, h->device) != cudaSuccess) {
        set_err(h, ENSC_ERR_CUDA, "cudaGetDeviceProperties failed");
        return fail(ENSC_ERR_CUDA);
    }
    const int occ_e = std::max(1, mx ? ensc::occupancy_element_mixed(h->plastic, ih.patch) : ensc::occupancy_element_fp64(h->plastic, ih.bt9));
    const int occ_n = std::max(1, mx ? ensc::occupancy_node_mixed() : ensc::occupancy_node_fp64());
    const int64_t ge = (h->ne + ensc::kElemThreads - 1) / ensc::kElemThreads;
    const int64_t node_threads = static_cast<int64_t>(ensc::kNodeThreads) * ensc::node_group_width(mx);
    const int64_t gn = (h->nn + node_threads - 1) / node_threads;
    h->grid_e = static_cast<int>(std::min<int64_t>(ge, static_cast<int64_t>(occ_e) * prop.multiProcessorCount));
    h->grid_n = static_cast<int>(std::min<int64_t>(gn, static_cast<int64_t>(occ_n) * prop.multiProcessorCount));

    // resident runs where the mesh fits on chip (slot assembly)
    if (!ih.patch && prop.cooperativeLaunch)
        h->run = mx ? ensc::plan_run_mixed(h->ne, h->nn, h->plastic, prop.multiProcessorCount)
                    : ensc::plan_run_fp64(h->ne, h->nn, h->plastic, ih.bt9, prop.multiProcessorCount);

    // ---- device memory: the instance block plus partial sums and control ----
    // (one partial slot per block of the larger of the two launch forms)
    const int pe = std::max(h->grid_e, h->run.grid), pn = std::max(h->grid_n, h->run.grid);
    const size_t pbytes = (3 * static_cast<size_t>(pe) + 2 * static_cast<size_t>(pn)) * sizeof(double);
    const size_t poff = (pbytes + 255) / 256 * 256, coff = (sizeof(Ctl) + 255) / 256 * 256;
    const size_t small = poff + coff + (sizeof(ensc::RunSync) + 255) / 256 * 256;
    cudaError_t ce = cudaMalloc(&h->arena, ih.bytes + small);
    if (ce != cudaSuccess) {
        cuda_err(h, "cudaMalloc(instance)", ce);
        return fail(ENSC_ERR_OOM);
    }
    h->arena_bytes = ih.bytes + small;
    if (cudaMallocHost(reinterpret_cast<void**>(&h->ctl_host), sizeof(Ctl)) != cudaSuccess) {
        set_err(h, ENSC_ERR_OOM, "cudaMallocHost(ctl)");
        return fail(ENSC_ERR_OOM);
    }
    if (params->stream) {
        h->stream = static_cast<cudaStream_t>(params->stream);
    } else {
        ce = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
        if (ce != cudaSuccess) {
            cuda_err(h, "cudaStreamCreate", ce);
            return fail(ENSC_ERR_CUDA);
        }
        h->own_stream = true;
    }
    ce = cudaStreamCreateWithFlags(&h->cap_stream, cudaStreamNonBlocking);
    if (ce != cudaSuccess) {
        cuda_err(h, "cudaStreamCreate(capture)", ce);
        return fail(ENSC_ERR_CUDA);
    }
    rc = ensc::instance_upload(ih, h->arena, h->stream, h->E, h->N, h->PA, perr);
    if (rc) {
        set_err(h, rc, perr);
        return fail(rc);
    }
    h->n_patches = ih.n_patches;
    h->n_partials = ih.n_pnodes;
    char* tail = static_cast<char*>(h->arena) + ih.bytes;
    h->P.elem = reinterpret_cast<double*>(tail);
    h->P.node = h->P.elem + 3 * pe;
    h->P.n_elem_blocks = pe;
    h->P.n_node_blocks = pn;
    h->ctl = reinterpret_cast<Ctl*>(tail + poff);
    h->sync = reinterpret_cast<ensc::RunSync*>(tail + poff + coff);
    ce = cudaMemsetAsync(tail, 0, small, h->stream);
    ensc::RunSync sync0{};
    sync0.pre = ensc::kInfBits;
    for (ensc::RunMins& m : sync0.mins) m = ensc::RunMins{ensc::kInfBits, ensc::kInfBits};
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(h->sync, &sync0, sizeof(sync0), cudaMemcpyHostToDevice, h->stream);
    if (ce != cudaSuccess) {
        cuda_err(h, "cudaMemset(partials)", ce);
        return fail(ENSC_ERR_CUDA);
    }
    // staging for AoS up/download: reuse the element force scratch when large enough
    const size_t need_stage = std::max<size_t>(12 * h->ne, 3 * h->nn) * sizeof(double);
    if (ih.size[ensc::InstanceHost::FE] >= need_stage) {
        h->staging = static_cast<double*>(h->E.fe);
    } else {
        ce = cudaMalloc(reinterpret_cast<void**>(&h->staging), need_stage);
        if (ce != cudaSuccess) {
            cuda_err(h, "cudaMalloc(staging)", ce);
            return fail(ENSC_ERR_OOM);
        }
        h->staging_owned = true;
    }
    h->staging_bytes = need_stage;

    ensc::material_from(mat, params, h->M);
    *h->ctl_host = ensc::initial_ctl(params, h->M);
    ce = cudaMemcpyAsync(h->ctl, h->ctl_host, sizeof(Ctl), cudaMemcpyHostToDevice, h->stream);
    if (ce != cudaSuccess) {
        cuda_err(h, "upload ctl", ce);
        return fail(ENSC_ERR_CUDA);
    }
    // init(): the force pass with dt = 0 and no boundary conditions, which
    // leaves the minimum element dt for the first cycle in ctl->dts_next
    launch_element(h, true, h->stream);
    ce = cudaGetLastError();
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(h->stream);
    if (ce != cudaSuccess) {
        cuda_err(h, "init pass", ce);
        return fail(ENSC_ERR_CUDA);
    }
    if (!h->run.grid) {
        rc = build_graph(h);
        if (rc) return fail(rc);
    }
    *out = h;
    return ENSC_OK;
}

int ensc_set_bcs(ensc_handle* h, const int8_t* dof_code, const double* dof_value) {
    if (!h) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    std::vector<uint8_t> bc;
    std::vector<double> bcv;
    ensc::pack_bcs(h->nn, h->nn_pad, dof_code, dof_value, bc, bcv);
    int rc = upload(h, const_cast<uint8_t*>(h->N.bc), bc);
    if (!rc && !bcv.empty()) rc = upload(h, const_cast<double*>(h->N.bcv), bcv);
    if (rc) return rc;
    ensc::launch_apply_bc_v(h->N, mixed(h), h->stream);
    if (!h->kinetic0_done) {
        if (int rs = settle_energy(h)) return rs;  // cycles may have run before the first conditions
        ensc::launch_kinetic0(h->N, h->P, h->ctl, mixed(h), h->grid_n, h->stream);
        h->kinetic0_done = true;
    }
    CK(h, cudaGetLastError());
    CK(h, cudaStreamSynchronize(h->stream));
    return ENSC_OK;
}

int ensc_set_gravity(ensc_handle* h, int32_t on, double value, const double dir[3]) {
    if (!h) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    h->M.gravity_on = on;
    h->M.gravity_value = value;
    for (int i = 0; i < 3; ++i) h->M.gravity_dir[i] = dir ? dir[i] : 0.0;
    return loads_changed(h);
}

int ensc_set_gravity_amplitude(ensc_handle* h, int32_t n_points, const double* time_value) {
    if (!h) return ENSC_ERR_ARG;
    if (n_points < 0 || n_points > ENSC_MAX_AMPLITUDE_POINTS || (n_points > 0 && !time_value))
        return set_err(h, ENSC_ERR_ARG, "amplitude: 0 to ENSC_MAX_AMPLITUDE_POINTS (time, value) pairs");
    DevGuard dg(h->device);
    if (n_points == 0) {
        h->M.amp = nullptr;
        h->M.amp_n = 0;
        return loads_changed(h);
    }
    if (!h->amp) {
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&h->amp), 2 * sizeof(double) * ENSC_MAX_AMPLITUDE_POINTS);
        if (e != cudaSuccess) {
            h->amp = nullptr;
            return cuda_err(h, "cudaMalloc(amplitude)", e);
        }
    }
    // stream order: cycles already enqueued finish with the previous table
    CK(h, cudaMemcpyAsync(h->amp, time_value, 2 * sizeof(double) * n_points, cudaMemcpyHostToDevice, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    h->M.amp = h->amp;
    h->M.amp_n = n_points;
    return loads_changed(h);
}

int ensc_step_async(ensc_handle* h, int64_t max_cycles, double step_end_time) {
    if (!h || max_cycles < 0) return ENSC_ERR_ARG;
    if (max_cycles == 0) return ENSC_OK;
    DevGuard dg(h->device);
    return enqueue_cycles(h, max_cycles, true, max_cycles, step_end_time, HUGE_VAL);
}

int ensc_step_until_async(ensc_handle* h, int64_t max_cycles, double step_end_time, double pause_time) {
    if (!h || max_cycles < 0) return ENSC_ERR_ARG;
    if (max_cycles > (int64_t(1) << 24))
        return set_err(h, ENSC_ERR_ARG, "ensc_step_until_async: at most 2^24 cycles per call");
    if (max_cycles == 0) return ENSC_OK;
    DevGuard dg(h->device);
    return enqueue_cycles(h, max_cycles, true, max_cycles, step_end_time, pause_time);
}

int ensc_sync(ensc_handle* h, ensc_step_report* report) {
    if (!h) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    const int64_t before = h->ctl_host->cycles_done;
    int rc = read_ctl(h);
    if (rc) return rc;
    fill_report(h, before, report);
    return status_code(h, h->ctl_host->status);
}

int ensc_step(ensc_handle* h, int64_t max_cycles, double step_end_time, ensc_step_report* report) {
    return ensc_step_until(h, max_cycles, step_end_time, HUGE_VAL, report);
}

int ensc_step_until(ensc_handle* h, int64_t max_cycles, double step_end_time, double pause_time,
                    ensc_step_report* report) {
    if (!h || max_cycles < 0) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    const int64_t before = h->ctl_host->cycles_done;
    if (max_cycles == 0) {
        int rc = read_ctl(h);
        if (rc) return rc;
    }
    // launch in batches; after each, the control block tells whether the call
    // is over (step end or pause reached, cycles spent, or a status)
    const int64_t batch = (kRunCycles + h->chunk - 1) / h->chunk * h->chunk;
    for (int64_t launched = 0; launched < max_cycles;) {
        const int64_t n = std::min(batch, max_cycles - launched);
        int rc = enqueue_cycles(h, n, launched == 0, max_cycles, step_end_time, pause_time);
        if (!rc) rc = read_ctl(h);
        if (rc) return rc;
        launched += n;
        if (h->ctl_host->done || h->ctl_host->status) break;
    }
    fill_report(h, before, report);
    return status_code(h, h->ctl_host->status);
}

// The staging area may be the element force scratch, whose slots no
// element fills must read as zeros for the node pass: clear what was used.
static int release_staging(ensc_handle* h, size_t used) {
    if (!h->staging_owned && used) {
        h->fe_valid = false;
        CK(h, cudaMemsetAsync(h->staging, 0, used, h->stream));
    }
    return ENSC_OK;
}

int ensc_download(ensc_handle* h, double* x, double* u, double* v, double* sigma, double* qia, double* eps_p) {
    if (!h) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    struct Item {
        double* dst;
        const void* rows;   // element rows, or null: a node field
        ensc::NodeField field;
        int64_t n;
        int comps;
    };
    using F = ensc::NodeField;
    const bool mx = mixed(h);
    const Item items[] = {{x, nullptr, F::X, h->nn, 3},          {u, nullptr, F::U, h->nn, 3},
                          {v, nullptr, F::V, h->nn, 3},          {sigma, h->E.sigma, F::X, h->ne, 6},
                          {qia, h->E.qia, F::X, h->ne, 12},      {eps_p, h->E.eps_p, F::X, h->ne, 1}};
    size_t used = 0;
    for (const Item& it : items) {
        if (!it.dst) continue;
        if (!it.rows) ensc::launch_nodes_to_aos(h->N, it.field, mx, h->staging, h->stream);
        else  // element fields, at their stored positions
            ensc::launch_elem_to_aos(h->E, it.rows, it.comps, mx, h->staging, h->stream, h->PA.iperm);
        CK(h, cudaGetLastError());
        CK(h, cudaMemcpyAsync(it.dst, h->staging, it.n * it.comps * sizeof(double), cudaMemcpyDeviceToHost,
                              h->stream));
        CK(h, cudaStreamSynchronize(h->stream));
        used = std::max(used, static_cast<size_t>(it.n * it.comps) * sizeof(double));
    }
    return release_staging(h, used);
}

int ensc_download_reactions(ensc_handle* h, double* rf) {
    if (!h || !rf) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    ensc::launch_reactions_to_aos(h->N, h->staging, h->stream);
    CK(h, cudaGetLastError());
    CK(h, cudaMemcpyAsync(rf, h->staging, h->nn * 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    return release_staging(h, static_cast<size_t>(h->nn * 3) * sizeof(double));
}

int ensc_upload_state(ensc_handle* h, const double* x, const double* u, const double* v, const double* sigma,
                      const double* qia, const double* eps_p, double time, double dt_i, double dt_i_1,
                      double dt_stable_min) {
    if (!h) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    struct Item {
        const double* src;
        void* rows;         // element rows, or null: a node field
        ensc::NodeField field;
        int64_t n;
        int comps;
    };
    using F = ensc::NodeField;
    const bool mx = mixed(h);
    const Item items[] = {{x, nullptr, F::X, h->nn, 3},          {u, nullptr, F::U, h->nn, 3},
                          {v, nullptr, F::V, h->nn, 3},          {sigma, h->E.sigma, F::X, h->ne, 6},
                          {qia, h->E.qia, F::X, h->ne, 12},      {eps_p, h->E.eps_p, F::X, h->ne, 1}};
    size_t used = 0;
    // mixed: the u rows hold x - u; they hold u while x and u are replaced
    const bool uref = mx && (x || u);
    if (uref) ensc::launch_reflect_rows(h->N, h->stream);
    cudaError_t ue = cudaGetLastError();
    const char* what = "ensc_upload_state";
    for (const Item& it : items) {
        if (!it.src || ue != cudaSuccess) continue;
        ue = cudaMemcpyAsync(h->staging, it.src, it.n * it.comps * sizeof(double), cudaMemcpyHostToDevice,
                             h->stream);
        if (ue != cudaSuccess) {
            what = "cudaMemcpyAsync(state upload)";
            break;
        }
        if (!it.rows) ensc::launch_aos_to_nodes(h->staging, h->N, it.field, mx, h->stream);
        else ensc::launch_aos_to_elem(h->staging, h->E, it.comps, it.rows, mx, h->stream, h->PA.iperm);
        ue = cudaGetLastError();
        used = std::max(used, static_cast<size_t>(it.n * it.comps) * sizeof(double));
    }
    // back to x - u in the u rows, also when an upload above failed
    if (uref) ensc::launch_reflect_rows(h->N, h->stream);
    if (ue == cudaSuccess) ue = cudaGetLastError();
    if (ue != cudaSuccess) {
        release_staging(h, used);
        return cuda_err(h, what, ue);
    }
    if (int rc0 = release_staging(h, used)) return rc0;
    int rc = read_ctl(h);
    if (rc) return rc;
    h->ctl_host->time = time;
    h->ctl_host->dt_i = dt_i;
    h->ctl_host->dt_i_1 = dt_i_1;
    if (dt_stable_min > 0.0) {
        long long b;
        std::memcpy(&b, &dt_stable_min, sizeof b);
        h->ctl_host->dts_next = static_cast<unsigned long long>(b);
    }
    CK(h, cudaMemcpyAsync(h->ctl, h->ctl_host, sizeof(Ctl), cudaMemcpyHostToDevice, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    return ENSC_OK;
}

int ensc_snapshot_begin(ensc_handle* h) {
    if (!h) return ENSC_ERR_ARG;
    if (!h->fe_valid)
        return set_err(h, ENSC_ERR_ARG,
                       "ensc_snapshot_begin: no force pass since the last download or upload; run a cycle first");
    DevGuard dg(h->device);
    const size_t nodes3 = static_cast<size_t>(3 * h->nn), elems6 = static_cast<size_t>(6 * h->ne);
    const size_t fields = (5 * nodes3 + elems6) * sizeof(double);
    if (!h->snap_dev) {
        h->snap_bytes = (fields + 255) / 256 * 256 + sizeof(Ctl);
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&h->snap_dev), h->snap_bytes);
        if (e != cudaSuccess) {
            h->snap_dev = nullptr;
            return cuda_err(h, "cudaMalloc(snapshot)", e);
        }
        for (int k = 0; k < 2; ++k) {
            e = cudaMallocHost(reinterpret_cast<void**>(&h->snap_host[k]), h->snap_bytes);
            if (e != cudaSuccess) {
                h->snap_host[k] = nullptr;
                return cuda_err(h, "cudaMallocHost(snapshot)", e);
            }
        }
        CK(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
        CK(h, cudaEventCreateWithFlags(&h->snap_captured, cudaEventDisableTiming));
        for (int k = 0; k < 2; ++k) CK(h, cudaEventCreateWithFlags(&h->snap_landed[k], cudaEventDisableTiming));
    }
    // the previous snapshot's copy to the host reads the device buffer this
    // one overwrites (the copy before it used the same host buffer and ran
    // earlier on the same copy stream)
    if (h->snap_count > 0) CK(h, cudaStreamWaitEvent(h->stream, h->snap_landed[(h->snap_count - 1) % 2], 0));
    double* d = h->snap_dev;
    const bool mx = mixed(h);
    if (mx) ensc::launch_acceleration_mixed(h->E, h->N, h->M, h->ctl, d + 3 * nodes3, h->stream, h->PA);
    else ensc::launch_acceleration_fp64(h->E, h->N, h->M, h->ctl, d + 3 * nodes3, h->stream);
    ensc::launch_nodes_to_aos(h->N, ensc::NodeField::X, mx, d, h->stream);
    ensc::launch_nodes_to_aos(h->N, ensc::NodeField::U, mx, d + nodes3, h->stream);
    ensc::launch_nodes_to_aos(h->N, ensc::NodeField::V, mx, d + 2 * nodes3, h->stream);
    ensc::launch_reactions_to_aos(h->N, d + 4 * nodes3, h->stream);
    ensc::launch_elem_to_aos(h->E, h->E.sigma, 6, mx, d + 5 * nodes3, h->stream, h->PA.iperm);
    CK(h, cudaGetLastError());
    char* ctl_copy = reinterpret_cast<char*>(d) + (h->snap_bytes - sizeof(Ctl));
    CK(h, cudaMemcpyAsync(ctl_copy, h->ctl, sizeof(Ctl), cudaMemcpyDeviceToDevice, h->stream));
    CK(h, cudaEventRecord(h->snap_captured, h->stream));
    const int k = static_cast<int>(h->snap_count % 2);
    CK(h, cudaStreamWaitEvent(h->copy_stream, h->snap_captured, 0));
    CK(h, cudaMemcpyAsync(h->snap_host[k], h->snap_dev, h->snap_bytes, cudaMemcpyDeviceToHost, h->copy_stream));
    CK(h, cudaEventRecord(h->snap_landed[k], h->copy_stream));
    h->snap_count += 1;
    return ENSC_OK;
}

int ensc_snapshot_wait(ensc_handle* h, ensc_snapshot* out) {
    if (!h || !out) return ENSC_ERR_ARG;
    if (h->snap_count == 0) return set_err(h, ENSC_ERR_ARG, "ensc_snapshot_wait: no snapshot begun");
    DevGuard dg(h->device);
    const int k = static_cast<int>((h->snap_count - 1) % 2);
    CK(h, cudaEventSynchronize(h->snap_landed[k]));
    const double* b = h->snap_host[k];
    const size_t nodes3 = static_cast<size_t>(3 * h->nn);
    out->x = b;
    out->u = b + nodes3;
    out->v = b + 2 * nodes3;
    out->a = b + 3 * nodes3;
    out->rf = b + 4 * nodes3;
    out->sigma = b + 5 * nodes3;
    Ctl c;
    std::memcpy(&c, reinterpret_cast<const char*>(b) + (h->snap_bytes - sizeof(Ctl)), sizeof(Ctl));
    out->time = c.time;
    out->dt_i = c.dt_i;
    out->dt_i_1 = c.dt_i_1;
    out->total_cycles = c.cycles_done;
    out->status = (c.status & ensc::ST_TIMEOUT) ? ENSC_ERR_TIMEOUT
                  : (c.status & ensc::ST_INVERTED) ? ENSC_ERR_INVERTED
                  : c.status ? ENSC_ERR_NONFINITE : ENSC_OK;
    return ENSC_OK;
}

int ensc_energy(ensc_handle* h, ensc_energy_report* out) {
    if (!h || !out) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    ensc::launch_between(h->ctl, h->P, 1, h->stream);
    CK(h, cudaGetLastError());
    int rc = read_ctl(h);
    if (rc) return rc;
    const double* e = h->ctl_host->energy;
    out->kinetic = e[0];
    out->internal = e[1];
    out->hourglass = e[2];
    out->viscous = e[3];
    out->external = e[4];
    out->kinetic0 = e[5];
    return ENSC_OK;
}

int ensc_profile(ensc_handle* h, int64_t max_cycles, double step_end_time, double ms[5], int64_t launches[5]) {
    if (!h || max_cycles < 0 || !ms || !launches) return ENSC_ERR_ARG;
    DevGuard dg(h->device);
    for (int i = 0; i < 5; ++i) {
        ms[i] = 0.0;
        launches[i] = 0;
    }
    cudaEvent_t ev[6];
    for (int i = 0; i < 6; ++i) CK(h, cudaEventCreate(&ev[i]));
    if (h->run.grid)
        if (int rs = settle_energy(h)) return rs;
    ensc::launch_arm(h->ctl, step_end_time, max_cycles, h->stream);
    int rc = ENSC_OK;
    for (int64_t c = 0; c < max_cycles && rc == ENSC_OK; ++c) {
        cudaEventRecord(ev[0], h->stream);
        ensc::launch_between(h->ctl, h->P, 0, h->stream);
        cudaEventRecord(ev[1], h->stream);
        ensc::launch_edge_prepass(h->E, h->N, h->ctl, h->grid_e, h->stream);
        cudaEventRecord(ev[2], h->stream);
        cudaEventRecord(ev[3], h->stream);  // begin_exact runs inside the prepass
        launch_element(h, false, h->stream);
        cudaEventRecord(ev[4], h->stream);
        launch_node(h, h->stream);
        cudaEventRecord(ev[5], h->stream);
        cudaError_t e = cudaEventSynchronize(ev[5]);
        if (e != cudaSuccess) {
            rc = cuda_err(h, "ensc_profile", e);
            break;
        }
        for (int k = 0; k < 5; ++k) {
            float t = 0.f;
            cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
            ms[k] += t;
            launches[k] += 1;
        }
        if (read_ctl(h) != ENSC_OK) break;
        if (h->ctl_host->done) break;
    }
    for (int i = 0; i < 6; ++i) cudaEventDestroy(ev[i]);
    return rc;
}

int64_t ensc_device_bytes(const ensc_handle* h) {
    if (!h) return 0;
    return static_cast<int64_t>(h->arena_bytes + (h->staging_owned ? h->staging_bytes : 0));
}

int32_t ensc_kernels_per_cycle(const ensc_handle* h) { return h && !h->run.grid ? 4 : 0; }

int ensc_assembly(const ensc_handle* h, int32_t* assembly, int64_t* patches, int64_t* partials) {
    if (!h) return ENSC_ERR_ARG;
    if (assembly) *assembly = h->PA.pf ? ENSC_ASSEMBLY_PATCH : ENSC_ASSEMBLY_SLOT;
    if (patches) *patches = h->n_patches;
    if (partials) *partials = h->n_partials;
    return ENSC_OK;
}

void ensc_destroy(ensc_handle* h) {
    if (!h) return;
    DevGuard dg(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->graph) cudaGraphExecDestroy(h->graph);
    if (h->cap_stream) cudaStreamDestroy(h->cap_stream);
    if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
    if (h->staging_owned && h->staging) cudaFree(h->staging);
    if (h->arena) cudaFree(h->arena);
    if (h->amp) cudaFree(h->amp);
    if (h->copy_stream) {
        cudaStreamSynchronize(h->copy_stream);
        cudaStreamDestroy(h->copy_stream);
    }
    if (h->snap_captured) cudaEventDestroy(h->snap_captured);
    for (int k = 0; k < 2; ++k) {
        if (h->snap_landed[k]) cudaEventDestroy(h->snap_landed[k]);
        if (h->snap_host[k]) cudaFreeHost(h->snap_host[k]);
    }
    if (h->snap_dev) cudaFree(h->snap_dev);
    if (h->ctl_host) cudaFreeHost(h->ctl_host);
    delete h;
}

}  // extern "C"
