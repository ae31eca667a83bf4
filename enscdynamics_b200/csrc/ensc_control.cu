// Cycle control and data-movement kernels.  Built with -fmad=false: the
// stable-time-step arithmetic reproduces the reference's
// update_minVertex_perMaterial_and_dt (Explicit3D/source/exDyna3D.cpp:663-686)
// and run()'s last-step clamp (:90-97) operation by operation.
#include "ensc_cycle.cuh"
#include "ensc_device.cuh"
#include "ensc_kernels.h"

#include <algorithm>
#include <cfloat>

namespace ensc {
namespace {

// Sums n values spaced by `stride` in a fixed order: thread t takes
// t, t+NT, t+2NT, ... left to right, then a fixed shared-memory tree.
__device__ double fixed_sum(const double* a, int n) {
    __shared__ double red[kCtlThreads];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += kCtlThreads) s = s + a[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kCtlThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + w];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

// Same fixed order over n values spaced by `stride`.
__device__ double fixed_sum_strided(const double* a, int n, int stride) {
    __shared__ double red[kCtlThreads];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += kCtlThreads) s = s + a[static_cast<int64_t>(i) * stride];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kCtlThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + w];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

// A warp's view of a control block: all of it in one trip to L2, scalar work on
// the copy by lane 0, and one trip back.  Read field by field, between the
// branches that need them, the same work took 7.7 us of a batch's cycle on
// B200 (2.9 us this way).
constexpr int kCtlWords = sizeof(Ctl) / 8;
static_assert(sizeof(Ctl) % 8 == 0 && kCtlWords <= 32, "a control block is one word per lane");
struct CtlCopy {
    union {
        Ctl c;
        unsigned long long w[kCtlWords];
    };
    __device__ CtlCopy() {}
    __device__ void load(const Ctl* g, int lane) {
        if (lane < kCtlWords) w[lane] = reinterpret_cast<const unsigned long long*>(g)[lane];
        __syncwarp();
    }
    __device__ void store(Ctl* g, int lane) {
        __syncwarp();
        if (lane < kCtlWords) reinterpret_cast<unsigned long long*>(g)[lane] = w[lane];
    }
};

// The first half of update_minVertex_perMaterial_and_dt for the next cycle:
// rotate dt_i_1 <- dt_i, advance time (computeSate :775-780) and fix dt_i_1
// unless the total-time clamp (:682-685) could fire, which needs this cycle's
// minimum element edge first (the edge prepass).  One warp.
__global__ void k_begin(Ctl* ctl) {
    cycle_kernel_enter();
    __shared__ CtlCopy s;
    s.load(ctl, threadIdx.x);
    if (s.c.done) return;
    __syncwarp();
    if (threadIdx.x == 0) {
        if (cycle_stops(&s.c, s.c.status)) s.c.done = 1;
        else cycle_begin(&s.c);
    }
    s.store(ctl, threadIdx.x);
}

// mode 1: fold the energy partials into the control block and clear the work
// partials, which accumulate over cycles between folds (the host folds
// before it reads energies); 2: fold as the initial kinetic energy.
__global__ void __launch_bounds__(kCtlThreads) k_between(Ctl* ctl, Partials P, int mode) {
    if (ctl->energy_pending || mode == 2) {
        const double ei = fixed_sum(P.elem + 0 * P.n_elem_blocks, P.n_elem_blocks);
        const double eh = fixed_sum(P.elem + 1 * P.n_elem_blocks, P.n_elem_blocks);
        const double ev = fixed_sum(P.elem + 2 * P.n_elem_blocks, P.n_elem_blocks);
        const double kin = fixed_sum(P.node + 0 * P.n_node_blocks, P.n_node_blocks);
        const double wx = fixed_sum(P.node + 1 * P.n_node_blocks, P.n_node_blocks);
        if (threadIdx.x == 0) {
            if (mode == 2) {
                ctl->energy[0] = kin;
                ctl->energy[5] = kin;
            } else {
                ctl->energy[0] = kin;
                ctl->energy[1] += ei;
                ctl->energy[2] += eh;
                ctl->energy[3] += ev;
                ctl->energy[4] += wx;
            }
            ctl->energy_pending = 0;
        }
        for (int i = threadIdx.x; i < 3 * P.n_elem_blocks; i += kCtlThreads) P.elem[i] = 0.0;
        for (int i = threadIdx.x; i < P.n_node_blocks; i += kCtlThreads) P.node[P.n_node_blocks + i] = 0.0;
    }
}

// Minimum squared edge of element e from the current coordinates.
__device__ __forceinline__ double element_edge_sq(const ElemArrays& E, const NodeArrays& N, int64_t e) {
    const uint32_t* cn = tile_row(E, E.conn, e) + (e & 31);
    const int64_t cs = tile_stride(E);
    double xyz[8][3];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t n = cn[k * cs];
#pragma unroll
        for (int c = 0; c < 3; ++c) xyz[k][c] = *node_x(N, c, n);
    }
    return min_edge_sq(xyz);
}

// Minimum element edge over the current coordinates (min_ele_edge,
// exDyna3D.cpp:1173-1220), needed before the element pass only in a cycle
// where the total-time clamp may fire; the last block then applies the clamp
// (begin_exact).
__global__ void __launch_bounds__(128) k_edge_prepass(ElemArrays E, NodeArrays N, Ctl* ctl) {
    cycle_kernel_enter();
    if (ctl->done || !ctl->need_exact) return;
    __shared__ unsigned long long red[4];
    double m = DBL_MAX;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < E.ne;
         e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const double mm = element_edge_sq(E, N, e);
        const double len = sqrt(mm);
        m = len < m ? len : m;
    }
    unsigned long long b = ord_bits(m);
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, b, o);
        b = w < b ? w : b;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long r = red[0];
        for (int i = 1; i < 4; ++i) r = red[i] < r ? red[i] : r;
        atomicMin(&ctl->len_min, r);
        // the last block to finish takes the edge minimum (through L2: this
        // block may hold an older copy) and begins the cycle (begin_exact)
        __threadfence();
        if (atomicAdd(&ctl->prepass_done, 1) == static_cast<int>(gridDim.x) - 1) {
            __threadfence();
            begin_exact(ctl, atomicOr(&ctl->len_min, 0ull));
            ctl->prepass_done = 0;
        }
    }
}


__global__ void k_arm(Ctl* ctl, double step_end, long long max_cycles, double pause) {
    ctl->step_end = step_end;
    ctl->pause_time = pause;
    ctl->cycles_target = ctl->cycles_done + max_cycles;
    ctl->done = 0;
}

// apply_boundary_condition_vec (exDyna3D.cpp:379-490): velocity conditions
// first, fixed DOFs last.
// One velocity component of a node: FP64, or the mixed stepper's float with
// its residual row.
template <typename VT>
__device__ __forceinline__ double load_v(const NodeArrays& N, int c, int64_t n) {
    if constexpr (sizeof(VT) == 4) return v_join(*node_vf(N, c, n), v_lo_rows(N.v, N.nn_pad)[c * N.nn_pad + n]);
    else return *node_v64(N, c, n);
}
template <typename VT>
__device__ __forceinline__ void store_v(const NodeArrays& N, int c, int64_t n, double v) {
    if constexpr (sizeof(VT) == 4) v_split(v, *node_vf(N, c, n), v_lo_rows(N.v, N.nn_pad)[c * N.nn_pad + n]);
    else *node_v64(N, c, n) = v;
}

template <typename VT>
__global__ void k_apply_bc_v(NodeArrays N) {
    for (int64_t n = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; n < N.nn;
         n += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const uint32_t code = N.bc[n];
        if (!code) continue;
        for (int c = 0; c < 3; ++c) {
            const uint32_t cc = (code >> (2 * c)) & 3u;
            if (cc & 2u) store_v<VT>(N, c, n, N.bcv[c * N.nn_pad + n]);
            if (cc & 1u) store_v<VT>(N, c, n, 0.0);
        }
    }
}

template <typename VT>
__global__ void __launch_bounds__(kNodeThreads) k_kinetic(NodeArrays N, Partials P) {
    double kin = 0.0;
    for (int64_t n = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; n < N.nn;
         n += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const double im = N.inv_mass[n];
        for (int c = 0; c < 3; ++c) {
            const double v = load_v<VT>(N, c, n);
            kin = kin + 0.5 * (v * v) / im;
        }
    }
    __shared__ double red[kNodeThreads];
    red[threadIdx.x] = kin;
    __syncthreads();
    for (int w = kNodeThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        P.node[blockIdx.x] = red[0];
        P.node[P.n_node_blocks + blockIdx.x] = 0.0;
    }
}

// Component c of entry s: rows of `pad` entries, or rows of 32 in tiles `tile`
// entries apart (the element arrays).
__device__ __forceinline__ int64_t row_entry(int64_t s, int c, int64_t pad, int64_t tile) {
    return tile ? (s >> 5) * tile + c * 32 + (s & 31) : c * pad + s;
}

// Entry e of the interleaved array is row position at[e] of the rows (at
// null: e).
template <typename ST>
__global__ void k_soa_to_aos(const ST* soa, int64_t n, int64_t pad, int64_t tile, int comps, const int32_t* at,
                             double* aos) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n * comps;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t e = i / comps;
        const int c = static_cast<int>(i - e * comps);
        aos[i] = static_cast<double>(soa[row_entry(at ? at[e] : e, c, pad, tile)]);
    }
}

// a <- x - a over the u rows: turns the reference position rows of a mixed
// instance into displacement rows and back
__global__ void k_reflect_rows(NodeArrays N) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < 3 * N.nn;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int c = static_cast<int>(i / N.nn);
        const int64_t n = i - c * N.nn, k = c * N.nn_pad + n;
        N.u[k] = *node_x(N, c, n) - N.u[k];
    }
}

// Node fields between interleaved xyz doubles and the device layout.
template <typename VT>
__global__ void k_nodes_to_aos(NodeArrays N, NodeField field, double* aos) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < 3 * N.nn;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t n = i / 3;
        const int c = static_cast<int>(i - 3 * n);
        if (field == NodeField::X) aos[i] = *node_x(N, c, n);
        else if (field == NodeField::V) aos[i] = load_v<VT>(N, c, n);
        else if (sizeof(VT) == 4) aos[i] = *node_x(N, c, n) - N.u[c * N.nn_pad + n];
        else aos[i] = *node_u64(N, c, n);
    }
}
template <typename VT>
__global__ void k_aos_to_nodes(const double* aos, NodeArrays N, NodeField field) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < 3 * N.nn;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t n = i / 3;
        const int c = static_cast<int>(i - 3 * n);
        if (field == NodeField::X) *node_x(N, c, n) = aos[i];
        else if (field == NodeField::V) store_v<VT>(N, c, n, aos[i]);
        else if (sizeof(VT) == 4) N.u[c * N.nn_pad + n] = aos[i];
        else *node_u64(N, c, n) = aos[i];
    }
}

template <typename DT>
__global__ void k_aos_to_soa(const double* aos, int64_t n, int64_t pad, int64_t tile, int comps, const int32_t* at,
                             DT* soa) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n * comps;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t e = i / comps;
        const int c = static_cast<int>(i - e * comps);
        soa[row_entry(at ? at[e] : e, c, pad, tile)] = static_cast<DT>(aos[i]);
    }
}

// ---- batched instances ---------------------------------------------------------
// Begins every instance's next cycle exactly as k_begin does for one
// instance (one warp per instance slot), after marking instances that have
// reached their limits as done, and counts the instances whose cycle needs
// the edge prepass.  The energy terms stay in the per-tile accumulators
// until k_fold_batch.  Each slot's element-pass scalars (dt_i_1, live) go to
// T.sparam; the edge prepass rewrites them where it decides dt.
__global__ void __launch_bounds__(128) k_begin_batch(BatchTables T, int begin) {
    // one warp per slot; the tables stay as they are while a batch steps
    __shared__ CtlCopy copies[4];
    const int lane = threadIdx.x & 31, slot = blockIdx.x * 4 + (threadIdx.x >> 5);
    const bool used = slot < T.counts[2];
    const int active = used ? T.desc[slot].active : 0;
    cycle_kernel_enter();
    if (!used) return;
    StageHdr h{0.0, 0, 0};
    if (active) {
        CtlCopy& s = copies[threadIdx.x >> 5];
        s.load(T.ctl + slot, lane);
        if (!s.c.done) {
            __syncwarp();
            if (lane == 0) {
                if (cycle_stops(&s.c, s.c.status)) {
                    s.c.done = 1;
                } else if (begin) {
                    cycle_begin(&s.c);
                    if (s.c.need_exact) atomicAdd(T.exact_count, 1);
                    h.dt1 = s.c.dt_i_1;
                    h.live = 1;
                }
            }
            s.store(T.ctl + slot, lane);
        }
    }
    if (lane == 0) T.sparam[slot] = h;
}

// Folds an instance's tile accumulators into its control block (one block
// per instance slot, tiles in order): the work terms are added and the tile
// accumulators cleared; the kinetic energy is the sum of the tiles' latest
// values when cycles ran since the last fold.
__global__ void __launch_bounds__(kCtlThreads) k_fold_batch(BatchTables T) {
    const int slot = blockIdx.x;
    if (slot >= T.counts[2]) return;
    const InstanceDesc& d = T.desc[slot];
    if (!d.active) return;
    Ctl* ctl = d.ctl;
    const int nw = T.etile / 32;  // element-tile partials: one per warp
    const int ne_part = d.e_ntiles * nw;
    double* ep = T.etile_part + 3 * static_cast<int64_t>(d.e_tile0) * nw;
    double* np = T.ntile_part + 2 * static_cast<int64_t>(d.n_tile0);
    const double ei = fixed_sum_strided(ep + 0, ne_part, 3);
    const double eh = fixed_sum_strided(ep + 1, ne_part, 3);
    const double ev = fixed_sum_strided(ep + 2, ne_part, 3);
    const double kin = fixed_sum_strided(np + 0, d.n_ntiles, 2);
    const double wx = fixed_sum_strided(np + 1, d.n_ntiles, 2);
    for (int i = threadIdx.x; i < 3 * ne_part; i += kCtlThreads) ep[i] = 0.0;
    for (int i = threadIdx.x; i < d.n_ntiles; i += kCtlThreads) np[2 * i + 1] = 0.0;
    if (threadIdx.x == 0) {
        if (ctl->energy_pending) ctl->energy[0] = kin;
        ctl->energy[1] += ei;
        ctl->energy[2] += eh;
        ctl->energy[3] += ev;
        ctl->energy[4] += wx;
        ctl->energy_pending = 0;
    }
}

// Minimum element edge for the instances whose cycle may hit the total-time
// clamp (see k_edge_prepass), one warp per element tile of T.etile elements.
__global__ void __launch_bounds__(128) k_edge_prepass_batch(BatchTables T) {
    cycle_kernel_enter();
    if (*T.exact_count == 0) return;
    const int lane = threadIdx.x & 31;
    const int warp = static_cast<int>((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
    const int nwarps = static_cast<int>((static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5);
    for (int t = warp; t < T.counts[0]; t += nwarps) {
        const InstanceDesc& d = T.desc[T.etile_inst[t]];
        Ctl* ctl = d.ctl;
        if (ctl->done || !ctl->need_exact) continue;
        const int64_t base = T.etile_base[t];
        const int64_t end = base + T.etile < d.E.ne ? base + T.etile : d.E.ne;
        double m = DBL_MAX;
        for (int64_t e = base + lane; e < end; e += 32) {
            const double mm = element_edge_sq(d.E, d.N, e);
            const double len = sqrt(mm);
            m = len < m ? len : m;
        }
        unsigned long long b = ord_bits(m);
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(0xffffffffu, b, o);
            b = w < b ? w : b;
        }
        if (lane == 0) atomicMin(&ctl->len_min, b);
    }
    // the last block to finish begins the exact cycles (k_begin_exact for
    // each such instance) and clears the counters
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(T.prepass_done, 1) == static_cast<int>(gridDim.x) - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int slot = threadIdx.x; slot < T.counts[2]; slot += blockDim.x) {
        const InstanceDesc& d = T.desc[slot];
        if (!d.active) continue;
        Ctl* ctl = d.ctl;
        if (ctl->done || !ctl->need_exact) continue;
        // the edge minimum through L2 (this block may hold an older copy)
        begin_exact(ctl, atomicOr(&ctl->len_min, 0ull));
        T.sparam[slot].dt1 = ctl->dt_i_1;
    }
    if (threadIdx.x == 0) {
        *T.prepass_done = 0;
        *T.exact_count = 0;
    }
}


int grid_for(int64_t work, int threads) {
    const int64_t g = (work + threads - 1) / threads;
    return static_cast<int>(g < 1 ? 1 : (g > 4096 ? 4096 : g));
}

}  // namespace

void launch_between_batch(const BatchTables& T, int slots, int mode, cudaStream_t st) {
    if (mode == 1) k_fold_batch<<<slots, kCtlThreads, 0, st>>>(T);
    launch_cycle_kernel(k_begin_batch, (slots + 3) / 4, 128, 0, st, T, mode == 0 ? 1 : 0);
}
void launch_edge_prepass_batch(const BatchTables& T, int grid, cudaStream_t st) {
    launch_cycle_kernel(k_edge_prepass_batch, grid, 128, 0, st, T);
}
void launch_between(Ctl* ctl, const Partials& P, int mode, cudaStream_t st) {
    if (mode == 0) launch_cycle_kernel(k_begin, 1, 32, 0, st, ctl);
    else k_between<<<1, kCtlThreads, 0, st>>>(ctl, P, mode);
}
void launch_edge_prepass(const ElemArrays& E, const NodeArrays& N, Ctl* ctl, int grid, cudaStream_t st) {
    launch_cycle_kernel(k_edge_prepass, grid, 128, 0, st, E, N, ctl);
}
void launch_arm(Ctl* ctl, double step_end, long long max_cycles, cudaStream_t st, double pause) {
    k_arm<<<1, 1, 0, st>>>(ctl, step_end, max_cycles, pause);
}
void launch_apply_bc_v(const NodeArrays& N, bool fp32_v, cudaStream_t st) {
    const int g = grid_for(N.nn, 256);
    if (fp32_v) k_apply_bc_v<float><<<g, 256, 0, st>>>(N);
    else k_apply_bc_v<double><<<g, 256, 0, st>>>(N);
}
void launch_kinetic0(const NodeArrays& N, const Partials& P, Ctl* ctl, bool fp32_v, int grid, cudaStream_t st) {
    if (fp32_v) k_kinetic<float><<<grid, kNodeThreads, 0, st>>>(N, P);
    else k_kinetic<double><<<grid, kNodeThreads, 0, st>>>(N, P);
    k_between<<<1, kCtlThreads, 0, st>>>(ctl, P, 2);
}
void launch_reactions_to_aos(const NodeArrays& N, double* aos, cudaStream_t st) {
    k_soa_to_aos<double><<<grid_for(3 * N.nn, 256), 256, 0, st>>>(N.rf, N.nn, N.nn_pad, 0, 3, nullptr, aos);
}
void launch_elem_to_aos(const ElemArrays& E, const void* rows, int comps, bool src_fp32, double* aos, cudaStream_t st,
                        const int32_t* at) {
    const int g = grid_for(E.ne * comps, 256);
    if (src_fp32)
        k_soa_to_aos<float><<<g, 256, 0, st>>>(static_cast<const float*>(rows), E.ne, 0, E.tile_bytes / 4, comps, at,
                                               aos);
    else
        k_soa_to_aos<double><<<g, 256, 0, st>>>(static_cast<const double*>(rows), E.ne, 0, E.tile_bytes / 8, comps, at,
                                                aos);
}
void launch_reflect_rows(const NodeArrays& N, cudaStream_t st) {
    k_reflect_rows<<<grid_for(3 * N.nn, 256), 256, 0, st>>>(N);
}
void launch_nodes_to_aos(const NodeArrays& N, NodeField field, bool mixed_precision, double* aos, cudaStream_t st) {
    const int g = grid_for(3 * N.nn, 256);
    if (mixed_precision) k_nodes_to_aos<float><<<g, 256, 0, st>>>(N, field, aos);
    else k_nodes_to_aos<double><<<g, 256, 0, st>>>(N, field, aos);
}
void launch_aos_to_nodes(const double* aos, const NodeArrays& N, NodeField field, bool mixed_precision,
                         cudaStream_t st) {
    const int g = grid_for(3 * N.nn, 256);
    if (mixed_precision) k_aos_to_nodes<float><<<g, 256, 0, st>>>(aos, N, field);
    else k_aos_to_nodes<double><<<g, 256, 0, st>>>(aos, N, field);
}
void launch_aos_to_elem(const double* aos, const ElemArrays& E, int comps, void* rows, bool dst_fp32, cudaStream_t st,
                        const int32_t* at) {
    const int g = grid_for(E.ne * comps, 256);
    if (dst_fp32)
        k_aos_to_soa<float><<<g, 256, 0, st>>>(aos, E.ne, 0, E.tile_bytes / 4, comps, at, static_cast<float*>(rows));
    else
        k_aos_to_soa<double><<<g, 256, 0, st>>>(aos, E.ne, 0, E.tile_bytes / 8, comps, at, static_cast<double*>(rows));
}

}  // namespace ensc
