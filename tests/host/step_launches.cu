// The host side of the step calls (csrc/ensc_capi.cu) against a CUDA runtime
// (fake_cudart.cpp) and kernels that are faked on the host: what is launched, and
// what is left in the partial sums.  A kernel is a function on a control block and
// partial sums in host memory.  Prints one line per scenario, read by
// test_step_launches.py.
#include "ensc_capi.cu"

#include "fake_cudart.h"

namespace {

int g_run_grid = 0;           // resident plan handed out at creation (0: none)
int g_refuse_run_after = -1;  // resident launches that succeed before one is refused
cudaError_t g_refusal = cudaErrorCooperativeLaunchTooLarge;
int g_singles = 0, g_runs = 0, g_arms = 0;
int64_t g_longest_run = 0;
constexpr int kGridN = 3;     // blocks of the fake node pass

void cycle_of(Ctl* c) {
    if (c->cycles_done >= c->cycles_target) c->done = 1;
}
// one cycle's kinetic energy: 1 + cycles_done, spread over the blocks of a grid
void fill_kinetic(const ensc::Partials& P, const Ctl* c, int grid) {
    for (int i = 0; i < grid; ++i) P.node[i] = (1.0 + c->cycles_done) / grid;
    P.elem[0] += 1.0;  // internal work: one unit a cycle
}

}  // namespace

// ---- kernels ----
namespace ensc {
void launch_between(Ctl* c, const Partials& P, int mode, cudaStream_t) {
    fake_launch([=] {
        if (mode == 0) {
            if (!c->done) cycle_of(c);
            return;
        }
        if (!c->energy_pending && mode != 2) return;
        double kin = 0.0, work = 0.0;
        for (int i = 0; i < P.n_node_blocks; ++i) kin += P.node[i];
        for (int i = 0; i < P.n_elem_blocks; ++i) work += P.elem[i];
        c->energy[0] = kin;
        if (mode == 2) c->energy[5] = kin;
        else c->energy[1] += work;
        for (int i = 0; i < 3 * P.n_elem_blocks; ++i) P.elem[i] = 0.0;
        c->energy_pending = 0;
    });
}
void launch_edge_prepass(const ElemArrays&, const NodeArrays&, Ctl*, int, cudaStream_t) {}
void launch_element_fp64(const ElemArrays&, const NodeArrays&, const Material&, Ctl*, const Partials&, int, bool,
                         cudaStream_t) {}
void launch_element_mixed(const ElemArrays&, const NodeArrays&, const Material&, Ctl*, const Partials&, int, bool,
                          cudaStream_t, const PatchArrays&) {}
void launch_node_fp64(const ElemArrays&, const NodeArrays&, const Material&, Ctl* c, const Partials& P, int grid,
                      cudaStream_t) {
    if (!fake_capturing()) g_singles += 1;
    fake_launch([=] {
        if (c->done) return;
        c->cycles_done += 1;
        c->energy_pending = 1;
        fill_kinetic(P, c, grid);
    });
}
void launch_node_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* c, const Partials& P, int grid,
                       cudaStream_t st, const PatchArrays&) {
    launch_node_fp64(E, N, M, c, P, grid, st);
}
void launch_arm(Ctl* c, double end, long long n, cudaStream_t, double pause) {
    g_arms += 1;
    c->step_end = end;
    c->pause_time = pause;
    c->cycles_target = c->cycles_done + n;
    c->done = 0;
}
cudaError_t launch_run_fp64(const RunPlan& p, const ElemArrays&, const NodeArrays&, const Material&, Ctl* c,
                            const Partials& P, RunSync*, const RunArgs& a, cudaStream_t st) {
    if (g_refuse_run_after >= 0 && g_runs >= g_refuse_run_after) return g_refusal;
    g_runs += 1;
    g_longest_run = std::max<int64_t>(g_longest_run, a.launch_cycles);
    if (a.arm) launch_arm(c, a.step_end, a.max_cycles, st, a.pause);
    for (int i = 0; i < a.launch_cycles && c->cycles_done < c->cycles_target; ++i) {
        c->cycles_done += 1;
        c->energy_pending = 1;
        fill_kinetic(P, c, p.grid);
    }
    cycle_of(c);
    return cudaSuccess;
}
cudaError_t launch_run_mixed(const RunPlan& p, const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* c,
                             const Partials& P, RunSync* s, const RunArgs& a, cudaStream_t st) {
    return launch_run_fp64(p, E, N, M, c, P, s, a, st);
}
void launch_kinetic0(const NodeArrays&, const Partials& P, Ctl* c, bool, int grid, cudaStream_t st) {
    for (int i = 0; i < grid; ++i) P.node[i] = 1.0 / grid;
    launch_between(c, P, 2, st);
}
RunPlan plan_run_fp64(int64_t, int64_t, bool, bool, int) {
    RunPlan p;
    p.grid = g_run_grid;
    p.threads = 128;
    p.tiles_per_warp = 1;
    return p;
}
RunPlan plan_run_mixed(int64_t a, int64_t b, bool c, int d) { return plan_run_fp64(a, b, c, true, d); }
int occupancy_element_fp64(bool, bool) { return 1; }
int occupancy_element_mixed(bool, bool) { return 1; }
int occupancy_node_fp64() { return 1; }
int occupancy_node_mixed() { return 1; }
int node_group_width(bool) { return 1; }
void launch_acceleration_fp64(const ElemArrays&, const NodeArrays&, const Material&, const Ctl*, double*, cudaStream_t) {}
void launch_acceleration_mixed(const ElemArrays&, const NodeArrays&, const Material&, const Ctl*, double*, cudaStream_t,
                               const PatchArrays&) {}
void launch_apply_bc_v(const NodeArrays&, bool, cudaStream_t) {}
void launch_nodes_to_aos(const NodeArrays&, NodeField, bool, double*, cudaStream_t) {}
void launch_aos_to_nodes(const double*, const NodeArrays&, NodeField, bool, cudaStream_t) {}
void launch_reactions_to_aos(const NodeArrays&, double*, cudaStream_t) {}
void launch_reflect_rows(const NodeArrays&, cudaStream_t) {}
void launch_elem_to_aos(const ElemArrays&, const void*, int, bool, double*, cudaStream_t, const int32_t*) {}
void launch_aos_to_elem(const double*, const ElemArrays&, int, void*, bool, cudaStream_t, const int32_t*) {}
int instance_prepare(const ensc_mesh_desc* m, const ensc_material*, bool mixed, int, InstanceHost& h, std::string&) {
    h.nn = m->n_nodes;
    h.ne = m->n_elements;
    h.nn_pad = (h.nn + 31) / 32 * 32;
    h.mixed = mixed;
    h.size[InstanceHost::FE] = 24 * 8 * static_cast<size_t>(h.nn_pad);
    h.bytes = h.size[InstanceHost::FE] + 4 * static_cast<size_t>(h.nn_pad);
    return ENSC_OK;
}
int instance_upload(const InstanceHost& h, void* block, cudaStream_t, ElemArrays& E, NodeArrays& N, PatchArrays&,
                    std::string&) {
    E.ne = h.ne;
    E.fe = block;
    N.nn = h.nn;
    N.nn_pad = h.nn_pad;
    N.bc = static_cast<uint8_t*>(block) + h.size[InstanceHost::FE];
    return ENSC_OK;
}
void pack_bcs(int64_t, int64_t pad, const int8_t*, const double*, std::vector<uint8_t>& bc, std::vector<double>& v) {
    bc.assign(static_cast<size_t>(pad), 0);
    v.clear();
}
void material_from(const ensc_material*, const ensc_params*, Material& M) { M = Material{}; }
Ctl initial_ctl(const ensc_params*, const Material&) { return Ctl{}; }
}  // namespace ensc

namespace {

ensc_handle* make(int run_grid, int chunk, int precision) {
    g_run_grid = run_grid;
    g_refuse_run_after = -1;
    g_singles = g_runs = g_arms = 0;
    fake_graph_launches() = 0;
    g_longest_run = 0;
    ensc_mesh_desc m{};
    m.n_nodes = kGridN * ensc::kNodeThreads;
    m.n_elements = 600;
    ensc_material mat{};
    ensc_params p{};
    p.precision = precision;
    p.factor_timestep = 0.7;
    p.graph_chunk = chunk;
    ensc_handle* h = nullptr;
    if (ensc_create(&m, &mat, &p, &h) != ENSC_OK) {
        printf("create failed: %s\n", ensc_last_error(nullptr));
        exit(1);
    }
    return h;
}
long long cycles(ensc_handle* h, int64_t n) {
    ensc_step_report r{};
    const int rc = ensc_step(h, n, 1e30, &r);
    return rc ? -1 : static_cast<long long>(r.total_cycles);
}

}  // namespace

int main() {
    // the split of a call on the per-phase kernels
    for (int chunk : {8, 32})
        for (int n : {1, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 4095, 4096, 4097, 4113}) {
            ensc_handle* h = make(0, chunk, ENSC_FP64);
            const long long c = cycles(h, n);
            printf("split %d %d %lld %d %d %d\n", chunk, n, c, fake_graph_launches(), g_singles, g_arms);
            ensc_destroy(h);
        }
    // resident calls: launches, and the longest of them
    for (int n : {1, 4096, 4097, 10000}) {
        ensc_handle* h = make(20, 32, ENSC_MIXED);
        const long long c = cycles(h, n);
        printf("resident %d %lld %d %lld %d %d\n", n, c, g_runs, static_cast<long long>(g_longest_run), fake_graph_launches(),
               g_singles);
        ensc_destroy(h);
    }
    // a launch that is refused, before any success and after `good` of them
    for (int precision : {ENSC_FP64, ENSC_MIXED})
        for (cudaError_t e : {cudaErrorCooperativeLaunchTooLarge, cudaErrorLaunchOutOfResources})
            for (int good : {0, 1, 2}) {
                ensc_handle* h = make(20, 32, precision);
                const int before = 7;
                for (int i = 0; i < good; ++i) cycles(h, before);
                g_refuse_run_after = g_runs;
                g_refusal = e;
                const long long c = cycles(h, 40);
                ensc_energy_report r{};
                ensc_energy(h, &r);
                printf("refused %d %lld %.17g %.17g %d\n", good, c, r.kinetic, r.internal,
                       static_cast<int>(ensc_kernels_per_cycle(h)));
                ensc_destroy(h);
            }
    return 0;
}
