// Resident runs: one launch that advances a single instance many cycles.
//
// A small or medium mesh spends its cycle on kernel boundaries: four launches
// a cycle, each with its drain, its gap and its cold start, take 18 us on
// B200 for 320 elements and 21 us for 27,556 (FP64), of which the element and
// node arithmetic is a few us.  Here the whole grid is resident, every warp
// keeps its element tiles (connectivity, geometry, sigma, QIA, eps_p) in
// shared memory from the first cycle to the last, and the element and node
// phases of each cycle are separated by barriers of the grid: a hardware
// cluster barrier where one cluster holds the mesh, else an arrival counter in
// global memory.  Node rows and element forces go through L2 as in the
// per-phase kernels.
//
// The scalar control (ensc_cycle.cuh) is evaluated by thread 0 of every block
// from the same values, so no block waits for another's decision.  The
// arithmetic per element and node is that of the per-phase kernels, and the
// minima are exact, so the state is bit-identical to theirs.
//
// Every wait on the counter and on a tile's copy is bounded (kStageWaitCycles);
// when one expires the block raises ST_TIMEOUT and leaves, and so do the others.
// The hardware barrier of a cluster has no limit of its own: all blocks of a
// cluster run at the same time, take the same decisions, and hold no wait
// without a limit between two of its barriers.
#pragma once

#include "ensc_cycle.cuh"
#include "ensc_device.cuh"
#include "ensc_kernels.h"
#include "ensc_stage.cuh"

#include <cfloat>

namespace ensc {

constexpr int kRunMaxWarps = 16;   // warps per block of a resident run
constexpr int kRunMaxCluster = 16;

struct RunShared {
    Ctl c;                         // thread 0's copy of the control block
    int32_t go, exact;
    double dt1, dt_i, dt_i_1, amp;
    int32_t cycles;                // cycles begun in this launch
    int32_t limit;                 // and the most that it may begin
    int32_t last;
    unsigned int bar;              // arrivals that complete the next barrier
    unsigned long long w_dts[kRunMaxWarps], w_len[kRunMaxWarps];
    // cluster barrier: what each block of the cluster published
    unsigned long long c_dts[kRunMaxCluster], c_len[kRunMaxCluster];
    int32_t c_bad[2][kRunMaxCluster];
    unsigned long long mbar[kRunMaxWarps];
};

__device__ __forceinline__ unsigned long long run_warp_min(unsigned long long v) {
    const unsigned hi = static_cast<unsigned>(v >> 32), lo = static_cast<unsigned>(v);
    const unsigned h = __reduce_min_sync(0xffffffffu, hi);
    const unsigned l = __reduce_min_sync(0xffffffffu, hi == h ? lo : 0xffffffffu);
    return (static_cast<unsigned long long>(h) << 32) | l;
}

// ---- batched element passes: a warp's sums over one tile ----
__device__ __forceinline__ double batch_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// The minima that a warp has sent to an instance's control block in this pass, in
// shared memory (lane 0's).  All tiles of a large instance would meet at two
// addresses there: a block of 2,097,152 elements alone in a batch took 326 us a
// cycle with two atomics per tile.
struct SentMinima {
    int32_t slot, pad;
    unsigned long long dts, len;
};
// Reduced per tile: between a warp's tiles, 100,000 elements and more apart, the
// instance changes almost always, and sums kept across tiles took the
// registers of the gathers.
__device__ __forceinline__ void batch_tile_sums(const BatchTables& T, int part, int slot, int lane, double ei,
                                                double eh, double ev, double dts, double len, int32_t bad,
                                                SentMinima* sent = nullptr) {
    ei = batch_warp_sum(ei);
    eh = batch_warp_sum(eh);
    ev = batch_warp_sum(ev);
    const unsigned long long dmin = run_warp_min(ord_bits(dts));
    const unsigned long long lmin = run_warp_min(ord_bits(len));
    bad = static_cast<int32_t>(__reduce_or_sync(0xffffffffu, static_cast<unsigned>(bad)));
    if (lane == 0) {
        // one writer per partial slot and pass: the reductions (no return
        // value) add in cycle order without a round trip
        double* p = T.etile_part + 3 * static_cast<int64_t>(part);
        Ctl* ctl = T.ctl + slot;
        atomicAdd(p + 0, ei);
        atomicAdd(p + 1, eh);
        atomicAdd(p + 2, ev);
        if (sent && sent->slot != slot) {
            sent->slot = slot;
            sent->dts = sent->len = kInfBits;
        }
        if (!sent || dmin < sent->dts) {
            atomicMin(&ctl->dts_next, dmin);
            if (sent) sent->dts = dmin;
        }
        if (!sent || lmin < sent->len) {
            atomicMin(&ctl->len_min, lmin);
            if (sent) sent->len = lmin;
        }
        if (bad) atomicOr(&ctl->status, bad);
    }
}

__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, unsigned long long v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ void st_cluster32(uint32_t addr, int32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// ---- barrier of the grid ----
// One thread per block, between block barriers: adds its arrival (the
// release covers what the block wrote before) and polls until `target`
// arrivals have been counted (the acquire covers what it reads after).
// Returns the counter as seen then, or all ones when the bounded wait
// expired.  With 148 blocks on B200 the bare barrier takes 2,460 clocks, two
// trips to L2 and back, and 3,460 behind 9 stores per thread.  Forms with a
// second hop (one collector that publishes, a tree of counters) took 3,100 to
// 4,350 bare; every block reading a table of all blocks, twice that.
__device__ __forceinline__ unsigned long long grid_barrier(unsigned long long* word, unsigned long long extra,
                                                           unsigned int target) {
    unsigned long long v;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(extra + 1ull) : "memory");
    const long long t0 = clock64();
    while (true) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
        if (static_cast<unsigned int>(v) >= target) return v;
        if (clock64() - t0 > kStageWaitCycles) return ~0ull;
    }
}
constexpr unsigned long long kRunErrElem = 1ull << 48, kRunErrNode = 1ull << 56;

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Thread 0 of every block, at the top of a cycle: stop, or begin the cycle.
__device__ __forceinline__ void run_begin(RunShared& sh, int32_t status, int launch_cycles) {
    Ctl* c = &sh.c;
    sh.go = 0;
    if (cycle_stops(c, status)) {
        c->done = 1;
        return;
    }
    if (sh.cycles >= launch_cycles) return;  // the rest in the next launch
    cycle_begin(c);
    sh.cycles += 1;
    sh.go = 1;
    sh.exact = c->need_exact;
    sh.dt1 = c->dt_i_1;
}

// The cycles of one launch.  Pol: the precision's element and node work.
//   Pol::kTileBytes                       bytes of one staged tile of 32 elements
//   Pol::load_tile(E, dst, bar, t, lane)      bulk copy of tile t
//   Pol::store_tile(E, tile, t, lane)         its evolving rows back to global memory
//   Pol::element(E, N, M, tile, dt1, e, lane, ...)
//   Pol::Nodes<W>                             a thread's W nodes: load (their rows), gather (their
//                                             forces), update
//   Pol::kinetic(N, n)                        kinetic energy of node n from its stored velocity
//   Pol::kKinInUpdate                         its velocities have more bits in the update than stored: the
//                                             kinetic energy is summed ahead of the last cycle's update
//                                             (Nodes::kinetic_after)
// Blocks of 32 * nw threads; warp w of the grid owns the tiles w, w + W, ...
template <class Pol, bool CLUSTER, int W>
__device__ __forceinline__ void run_cycles(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl,
                                           const Partials& P, RunSync* sync, const RunArgs& a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ RunShared sh;
    __shared__ double red[5][kRunMaxWarps];  // the warps' sums at the end of the launch
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    const int nblocks = gridDim.x, block = blockIdx.x;
    const int64_t ntiles = (E.ne + 31) / 32;
    const int64_t wstride = static_cast<int64_t>(nblocks) * nw;
    const int64_t w0 = static_cast<int64_t>(block) * nw + wid;
    const int mine = w0 < ntiles ? static_cast<int>((ntiles - 1 - w0) / wstride) + 1 : 0;
    unsigned char* wtiles = smem + static_cast<size_t>(wid) * a.tiles_per_warp * Pol::kTileBytes;

    if (tid == 0) {
        sh.c = *ctl;
        if (a.arm) {
            sh.c.step_end = a.step_end;
            sh.c.pause_time = a.pause;
            sh.c.cycles_target = sh.c.cycles_done + a.max_cycles;
            sh.c.done = 0;
        }
        sh.cycles = 0;
        const long long left = sh.c.cycles_target - sh.c.cycles_done;
        sh.limit = left < a.launch_cycles ? static_cast<int32_t>(left) : a.launch_cycles;
        sh.bar = 0;
        sh.go = 0;
        sh.exact = 0;
        if (!sh.c.done) run_begin(sh, sh.c.status, a.launch_cycles);
    }
    __syncthreads();
    if (!sh.go) {
        // nothing to run, in any block of the launch: only the limits and `done`
        // change, to the same values whichever of the old and new ones another
        // block reads
        if (tid == 0 && block == 0) *ctl = sh.c;
        return;
    }
    // another block's shared memory may be written once that block runs: every
    // block of a cluster arrives here, and waits before its first such store
    if (CLUSTER) cluster_arrive();
    bool loaded = true;
    if (mine > 0) {
        const uint32_t bar = smem_addr(&sh.mbar[wid]);
        if (lane == 0) {
            mbar_init(bar, mine);
            mbar_init_fence();
        }
        __syncwarp();
        for (int s = 0; s < mine; ++s)
            Pol::load_tile(E, smem_addr(wtiles + s * Pol::kTileBytes), bar, w0 + s * wstride, lane);
        loaded = mbar_wait_bounded(bar, 0);
        loaded = __all_sync(0xffffffffu, loaded);
    }
    if (CLUSTER) cluster_wait();
    double e_int = 0.0, e_hg = 0.0, e_vis = 0.0, wext = 0.0;
    const int64_t t0 = static_cast<int64_t>(block) * blockDim.x + tid;
    const int64_t stride = static_cast<int64_t>(nblocks) * blockDim.x;
    bool failed = false;
    bool ends = false;  // the cycle is the launch's last, unless an error makes an earlier one so
    int32_t err = 0;  // warp 0: an error was published
    while (sh.go) {
        const int set = sh.cycles % 3;
        if (sh.exact) {
            // a cycle the total-time clamp may shorten: the edge minimum first
            double m = DBL_MAX;
            for (int s = 0; s < mine && loaded; ++s) {
                if ((w0 + s * wstride) * 32 + lane >= E.ne) continue;
                const uint32_t* cn = Pol::conn(wtiles + s * Pol::kTileBytes);
                double xyz[8][3];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t n = cn[k * 32 + lane];
#pragma unroll
                    for (int c = 0; c < 3; ++c) xyz[k][c] = *node_x(N, c, n);
                }
                const double t = sqrt(min_edge_sq(xyz));
                m = t < m ? t : m;
            }
            const unsigned long long b = run_warp_min(ord_bits(m));
            if (lane == 0) sh.w_len[wid] = b;
            __syncthreads();
            unsigned long long l = kInfBits;
            if (wid == 0) {
                l = run_warp_min(lane < nw ? sh.w_len[lane] : kInfBits);
                if (CLUSTER) {
                    if (lane < nblocks) st_cluster(map_to_rank(smem_addr(&sh.c_len[block]), lane), l);
                } else if (lane == 0) {
                    atomicMin(&sync->pre, l);
                    sh.bar += nblocks;
                    if (grid_barrier(&sync->arrive, 0, sh.bar) == ~0ull) failed = true;
                    l = ld_relaxed(&sync->pre);
                }
            }
            if (CLUSTER) {
                cluster_arrive();
                cluster_wait();
            }
            if (wid == 0) {
                if (CLUSTER) l = run_warp_min(lane < nblocks ? sh.c_len[lane] : kInfBits);
                if (lane == 0) {
                    begin_exact(&sh.c, l);
                    sh.dt1 = sh.c.dt_i_1;
                }
            }
            if (CLUSTER) {
                // c_len is written again at the end of the element phase
                cluster_arrive();
                cluster_wait();
            }
            failed = __syncthreads_or(failed);
            if (failed) break;
        }
        // ---- element phase
        const double dt1 = sh.dt1;
        double dts_min = DBL_MAX, len_min = DBL_MAX;
        int32_t bad = loaded ? 0 : ST_TIMEOUT;
        for (int s = 0; s < mine && loaded; ++s) {
            const int64_t e = (w0 + s * wstride) * 32 + lane;
            if (e < E.ne) {
                double dts, len;
                Pol::element(E, N, M, wtiles + s * Pol::kTileBytes, dt1, e, lane, dts, len, e_int, e_hg, e_vis, bad);
                dts_min = dts < dts_min ? dts : dts_min;
                len_min = len < len_min ? len : len_min;
            }
        }
        if (bad) atomicOr(&sync->status, bad);
        {
            const unsigned long long d = run_warp_min(ord_bits(dts_min)), l = run_warp_min(ord_bits(len_min));
            if (lane == 0) {
                sh.w_dts[wid] = d;
                sh.w_len[wid] = l;
            }
        }
        int any_bad = __syncthreads_or(bad);
        if (wid == 0) {
            const unsigned long long d = run_warp_min(lane < nw ? sh.w_dts[lane] : kInfBits);
            const unsigned long long l = run_warp_min(lane < nw ? sh.w_len[lane] : kInfBits);
            if (CLUSTER) {
                if (lane < nblocks) {
                    st_cluster(map_to_rank(smem_addr(&sh.c_dts[block]), lane), d);
                    st_cluster(map_to_rank(smem_addr(&sh.c_len[block]), lane), l);
                    st_cluster32(map_to_rank(smem_addr(&sh.c_bad[0][block]), lane), any_bad);
                }
            } else if (lane == 0) {
                atomicMin(&sync->mins[set].dts, d);
                atomicMin(&sync->mins[set].len, l);
            }
        }
        // the thread's own node rows are on their way while the grid finishes
        typename Pol::template Nodes<W> nodes;
        if (CLUSTER) cluster_arrive();
        // (by every thread while it waits: decided by thread 0 along with dt, it took
        // 0.25 us of a 4.6 us cycle)
        if (Pol::kKinInUpdate)
            ends = !(sh.c.time < sh.c.step_end) | !(sh.c.time < sh.c.pause_time) | (sh.cycles >= sh.limit);
        nodes.load(E, N, M, t0);
        if (CLUSTER) {
            cluster_wait();
        } else {
            if (tid == 0) {
                sh.bar += nblocks;
                const unsigned long long v = grid_barrier(&sync->arrive, any_bad ? kRunErrElem : 0, sh.bar);
                if (v == ~0ull) failed = true;
                err |= static_cast<int32_t>((v >> 48) & 0xffu);
            }
            if (__syncthreads_or(failed)) {
                failed = true;
                ends = false;
                break;
            }
        }
        // the forces are added up while thread 0 turns the minima into dt
        unsigned long long d = 0, l = 0;
        if (!CLUSTER && tid == 0) {
            d = ld_relaxed(&sync->mins[set].dts);
            l = ld_relaxed(&sync->mins[set].len);
        }
        nodes.gather(E, N, M, t0);
        if (wid == 0) {
            if (CLUSTER) {
                d = run_warp_min(lane < nblocks ? sh.c_dts[lane] : kInfBits);
                l = run_warp_min(lane < nblocks ? sh.c_len[lane] : kInfBits);
                err |= __any_sync(0xffffffffu, lane < nblocks && sh.c_bad[0][lane] != 0);
            }
            if (lane == 0) {
                Ctl* c = &sh.c;
                c->dts_next = d;
                c->len_min = l;
                const double dt_i = cycle_dt(c, l, M.mc.inv_wos);
                if (!c->dt_final) c->dt_i = dt_i;
                c->cycles_done += 1;
                sh.dt_i = dt_i;
                sh.dt_i_1 = c->dt_i_1;
                sh.amp = (M.gravity_on && M.amp_n > 0) ? gravity_amplitude(M.amp, M.amp_n, c->time, dt_i) : 1.0;
                if (!(dt_i > 0.0) || !isfinite(dt_i)) {
                    err |= 1;
                    atomicOr(&sync->status, ST_BAD_DT);
                }
                if (!CLUSTER && block == 0) {
                    // the set of the next cycle restarts from +inf (its last
                    // readers passed the previous cycle's barriers)
                    sync->mins[(set + 1) % 3] = RunMins{kInfBits, kInfBits};
                    if (sh.exact) sync->pre = kInfBits;
                }
            }
        }
        __syncthreads();
        // ---- node phase
        int32_t nbad = 0;
        if constexpr (Pol::kKinInUpdate)
            if (ends) {
                const double k = batch_warp_sum(nodes.kinetic_after(E, N, M, sh.dt_i, sh.dt_i_1, sh.amp, t0, stride));
                if (lane == 0) red[4][wid] = k;
            }
        nodes.update(E, N, M, sh.dt_i, sh.dt_i_1, sh.amp, t0, stride, wext, nbad);
        if (nbad) atomicOr(&sync->status, nbad);
        any_bad = __syncthreads_or(nbad);
        if (CLUSTER) {
            if (tid < nblocks) st_cluster32(map_to_rank(smem_addr(&sh.c_bad[1][block]), tid), any_bad);
            cluster_arrive();
            cluster_wait();
        }
        if (wid == 0) {
            if (CLUSTER) {
                err |= __any_sync(0xffffffffu, lane < nblocks && sh.c_bad[1][lane] != 0);
            } else if (lane == 0) {
                sh.bar += nblocks;
                const unsigned long long v = grid_barrier(&sync->arrive, any_bad ? kRunErrNode : 0, sh.bar);
                if (v == ~0ull) failed = true;
                err |= static_cast<int32_t>(v >> 56);
            }
            if (lane == 0) run_begin(sh, err, a.launch_cycles);
        }
        if (__syncthreads_or(failed)) {
            failed = true;
            break;
        }
    }
    // ---- end of the launch: the evolving element rows, the energy partials
    // and the control block back to global memory
    for (int s = 0; s < mine && loaded; ++s)
        Pol::store_tile(E, wtiles + s * Pol::kTileBytes, w0 + s * wstride, lane);
    if (tid == 0 && failed) atomicOr(&sync->status, ST_TIMEOUT);
    // kinetic energy, unless the last cycle has summed it (a mixed run that an error
    // ended did not know its last cycle)
    double kin = 0.0;
    if (!ends)
        for (int64_t n = t0; n < N.nn; n += stride) kin = kin + Pol::kinetic(N, n);
    double v5[5] = {e_int, e_hg, e_vis, wext, kin};
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const double s = batch_warp_sum(v5[i]);
        if (lane == 0 && !(i == 4 && ends)) red[i][wid] = s;
    }
    __syncthreads();
    if (tid < 5) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s = s + red[tid][w];
        if (tid < 3) atomicAdd(P.elem + static_cast<int64_t>(tid) * P.n_elem_blocks + block, s);
        else if (tid == 3) atomicAdd(P.node + P.n_node_blocks + block, s);
        else
            // the latest kinetic energy: this run's blocks hold all of it
            for (int i = block; i < P.n_node_blocks; i += nblocks) P.node[i] = i == block ? s : 0.0;
    }
    // the last block out leaves the control block and a fresh sync area
    __threadfence();
    __syncthreads();
    if (tid == 0) sh.last = atomicAdd(&sync->left, 1) == nblocks - 1;
    __syncthreads();
    if (!sh.last || tid != 0) return;
    __threadfence();
    sh.c.status |= atomicExch(&sync->status, 0);
    sh.c.energy_pending = 1;
    *ctl = sh.c;
    for (int i = 0; i < 3; ++i) sync->mins[i] = RunMins{kInfBits, kInfBits};
    sync->pre = kInfBits;
    sync->arrive = 0;
    sync->left = 0;
}

// ---- host side ----
// Up to 4 warps per SM (one per scheduler) while that spreads the tiles over
// all SMs or fills one cluster; then more warps per block, then more tiles
// per warp, as far as shared memory goes.  A cluster's barrier takes about a
// third of the counter's, so it is used while 4 warps on each of its blocks
// hold the mesh.  Warps without a tile are added where they give every node
// a thread of its own (a node phase of 1,500 clocks against 3,600 with two
// nodes per thread, FP64 under gravity).
constexpr size_t kRunSmemMax = 227 * 1024 - sizeof(RunShared) - 5 * kRunMaxWarps * sizeof(double) - 256;

template <typename K>
RunPlan plan_run(K cluster_kernel_1, K cluster_kernel_2, K grid_kernel_1, K grid_kernel_2, int64_t ne, int64_t nn,
                 int sms, int max_warps, uint32_t tile_bytes) {
    RunPlan p;
    // one node per thread while there is a thread for every node
    auto width = [nn](const RunPlan& q) { return nn <= static_cast<int64_t>(q.grid) * q.threads ? 1 : 2; };
    sms = sms < 255 ? sms : 255;  // the error counts have 8 bits
    const int64_t tiles = (ne + 31) / 32;
    if (tiles <= 4 * kRunMaxCluster) {
        int c = 1;
        while (4 * c < tiles || (128 * c < nn && c < kRunMaxCluster)) c *= 2;
        p.threads = 128;
        p.grid = p.cluster = c;
        p.tiles_per_warp = 1;
        p.smem = static_cast<size_t>(4) * tile_bytes;
        p.node_width = width(p);
        K cluster_kernel = p.node_width == 1 ? cluster_kernel_1 : cluster_kernel_2;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(p.threads);
        cfg.dynamicSmemBytes = p.smem;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = c;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kRunSmemMax)) == cudaSuccess &&
            cudaFuncSetAttribute(cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&n, cluster_kernel, &cfg) == cudaSuccess && n > 0)
            return p;
        cudaGetLastError();
        p = RunPlan{};
    }
    p.grid = static_cast<int>(tiles < 4ll * sms ? (tiles + 3) / 4 : sms);
    int64_t w = (tiles + p.grid - 1) / p.grid;
    w = w < 4 ? 4 : (w > max_warps ? max_warps : w);
    const int64_t k = (tiles + p.grid * w - 1) / (p.grid * w);
    const int64_t wn = (nn + 32ll * p.grid - 1) / (32ll * p.grid);
    if (k == 1 && wn > w && wn <= max_warps) w = wn;
    p.threads = static_cast<int>(32 * w);
    const size_t need = static_cast<size_t>(w * k) * tile_bytes;
    p.node_width = width(p);
    K grid_kernel = p.node_width == 1 ? grid_kernel_1 : grid_kernel_2;
    int nb = 0;
    if (need > kRunSmemMax ||
        cudaFuncSetAttribute(grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kRunSmemMax)) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, grid_kernel, p.threads, need) != cudaSuccess || nb < 1) {
        cudaGetLastError();
        return RunPlan{};
    }
    p.tiles_per_warp = static_cast<int>(k);
    p.smem = need;
    return p;
}

// All blocks of the grid are resident at once: one cluster, or a cooperative
// launch.
template <typename K, typename... A>
cudaError_t launch_run(K kernel, const RunPlan& p, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.grid);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    if (p.cluster) {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = p.cluster;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace ensc
