// Device-side data structures shared by the stepper kernels.
//
// Memory layout in HBM:
//   element arrays: one tile of 32 consecutive elements after another
//   (ElemTile below); within a tile every component is a row of 32 entries, so
//   a warp of consecutive elements reads consecutive words, and a whole tile
//   is one contiguous copy.  Instances on caller-owned memory (ensc_step_noalloc) keep
//   plain rows of ne entries per component instead (tile_bytes 0).
//     conn[8] uint32                 local node k of the element
//     bt                             FP64: the 9 numbers the one-point B0^T
//                                    rows are formed from, or its 24 numbers
//                                    row-major (3*k + c); mixed: A as 9 hi and
//                                    9 lo floats
//     vol0, cbrt_v0, cbrt_v0sq       per-element constants
//     sigma[6], qia[12], eps_p
//     fe                             element nodal forces of the current cycle
//                                    (the element -> node hand-off, scratch):
//                                    by node and local slot when no node
//                                    repeats a slot, by node and row (rows) when
//                                    none has more than 8 elements, else by
//                                    element; per slot a row of (fx, fy) pairs, after the eight of
//                                    them a row of fz per slot (force_xy, force_z)
//   node arrays, length nn (stride nn_pad), in 32-byte records that one load
//   brings in (rec 1):
//     FP64:  x = [nn_pad] {x, y, z, ux}, u = [nn_pad] {uy, uz, vx, vy}, v = vz
//     mixed: x = [nn_pad] {x, y, z, (vx, vy) as two floats}, v = vz as float, then
//            the 16-bit residual rows [3][nn_pad] of v; u = [3][nn_pad] rows of
//            the reference position x - u
//     caller-owned memory (rec 0, FP64): plain rows [3][nn] of x, u and v
//     inv_mass[nn]                   per node (equal for the 3 DOFs)
//     bc[nn] uint8                   2 bits per DOF (bit0 fixed, bit1 velocity)
//     bcv[3][nn_pad]                 prescribed velocities
//     ell[8][nn] uint32              caller-owned memory: element holding node n
//                                    in local slot k, or ENSC_NONE; the gather sums
//                                    slots k = 0..7 in order, as the reference sums
//                                    its 8 slot vectors (exDyna3D.cpp:638-639)
//     csr_ptr/csr_ent                general (slot, element)-sorted lists, where
//                                    a node occupies the same slot in more than
//                                    one element and has more than 8 elements
#pragma once

#include <cmath>
#include <cstring>

#include <cstdint>
#include <cuda_runtime.h>

#define ENSC_NONE 0xFFFFFFFFu

namespace ensc {

// Status bits raised on the device and read back by the host.
enum : int32_t {
    ST_NONFINITE = 1,
    ST_INVERTED = 2,
    ST_BAD_DT = 4,       // stable dt not positive and finite
    ST_TIMEOUT = 8,      // a bounded wait for staged data expired; the pass stopped early
};

// Per-instance control block: the scalar state of exDyna3D's time loop
// (time, dt_i, dt_i_1: exDyna3D.h:175-178) plus the reductions that feed it.
struct Ctl {
    double time, dt_i, dt_i_1;
    double dt_prev;            // dt_i at the start of the cycle
    double step_end, total_time;
    double pause_time;         // stop after the cycle in which time reaches it (no dt clamp)
    double factor, wos;
    double dts_cur;            // min element dt of the previous force pass
    unsigned long long dts_next;   // ordered bits of min element dt, this pass
    unsigned long long len_min;    // ordered bits of min element edge, this pass
    long long cycles_done, cycles_target;
    int32_t done;
    int32_t need_exact;        // total-time clamp possible: edge minimum needed first
    int32_t dt_final;          // dt_i already fixed for this cycle
    int32_t energy_pending;    // partial energy sums of the last cycle not yet folded
    int32_t status;
    int32_t prepass_done;      // blocks of the edge prepass that have finished
    double energy[6];          // kinetic, internal, hourglass, viscous, external, kinetic0
};

// Constants of the mixed-precision element pass, derived once per instance
// on the host (set_mixed_consts).  lambda and 2G are float pairs (hi + lo);
// DRc and CRc are the per-element-invariant factors of the hourglass
// stiffness and damping; the element dt uses 1/wos and cvisq^2/wos in FP64.
struct MixedConsts {
    float G, lam_hi, lam_lo, g2_hi, g2_lo, rho, wos, cvisl, cvisq, y0, H, DRc, CRc, inv_3gh, pad[2];
    double inv_wos, cq2_wos;
};

struct Material {
    double E, nu, rho, G, K, lambda, wos;
    double yield0, hardening;
    double c_dr, c_cr, cvisl, cvisq;
    int32_t plastic;
    int32_t gravity_on;
    double gravity_value, gravity_dir[3];
    // gravity amplitude table: amp_n (time, value) pairs in device memory
    const double* amp;
    int32_t amp_n;
    MixedConsts mc;
};

// Fills M.mc from the FP64 material and controls; call after every change
// of them.
inline void set_mixed_consts(Material& M) {
    MixedConsts& c = M.mc;
    c = MixedConsts{};
    c.G = static_cast<float>(M.G);
    c.lam_hi = static_cast<float>(M.lambda);
    c.lam_lo = static_cast<float>(M.lambda - static_cast<double>(c.lam_hi));
    c.g2_hi = static_cast<float>(2.0 * M.G);
    c.g2_lo = static_cast<float>(2.0 * M.G - static_cast<double>(c.g2_hi));
    c.rho = static_cast<float>(M.rho);
    c.wos = static_cast<float>(M.wos);
    c.cvisl = static_cast<float>(M.cvisl);
    c.cvisq = static_cast<float>(M.cvisq);
    c.y0 = static_cast<float>(M.yield0);
    c.H = static_cast<float>(M.hardening);
    c.DRc = static_cast<float>(M.c_dr * (4.0 / 3.0 * M.G + M.K) * 0.1 / std::sqrt(8.0));
    c.CRc = static_cast<float>(M.c_cr * M.rho * M.wos / 4.0);
    c.inv_3gh = static_cast<float>(1.0 / (3.0 * M.G + M.hardening));
    c.inv_wos = 1.0 / M.wos;
    c.cq2_wos = M.cvisq * M.cvisq / M.wos;
}

// Byte offsets of the rows in a tile of 32 elements: what does not change
// first, then the evolving rows, eps_p last (elastic instances do not copy
// it).  The tile is copied to shared memory as it is.
template <typename Real, int kGeom, int kConsts>
struct ElemTile {
    static constexpr uint32_t kRow = 32u * sizeof(Real);
    static constexpr uint32_t kConn = 0;
    static constexpr uint32_t kBt = 8u * 32u * 4u;
    static constexpr uint32_t kVol0 = kBt + kGeom * kRow;          // doubles
    static constexpr uint32_t kCb = kVol0 + 32u * 8u;              // cbrt(V0) (FP64: and cbrt(V0^2))
    static constexpr uint32_t kState = kCb + kConsts * kRow;
    static constexpr uint32_t kSig = kState;
    static constexpr uint32_t kQia = kSig + 6u * kRow;
    static constexpr uint32_t kEps = kQia + 12u * kRow;
    static constexpr uint32_t kBytes = kEps + kRow;
};
using MixedTile = ElemTile<float, 18, 1>;    // 6,144 bytes
using Fp64Tile9 = ElemTile<double, 9, 2>;    // 8,960 bytes
using Fp64Tile24 = ElemTile<double, 24, 2>;  // 12,800 bytes

struct ElemArrays {
    int64_t ne, ne_pad;
    const uint32_t* conn;
    const void* bt;            // double (FP64) or float (mixed)
    const double* vol0;
    const void* cbrt_v0;       // double (FP64) or float (mixed)
    const double* cbrt_v0sq;   // FP64
    void* sigma;
    void* qia;
    void* eps_p;
    void* fe;
    // meshes whose nodes repeat local slots, with at most 8 elements at a node:
    // the row of fe that each local node's force goes to, 4 bits per local node
    // (null: the slot itself)
    const uint32_t* rows;
    // bytes of a tile of 32 elements; the pointers above point into tile 0,
    // which starts 256-byte aligned (node rows too, padded to 32 entries: the
    // vectorised node passes).  0: plain rows of ne_pad entries.
    int32_t tile_bytes;
    // 1: the entries of fe are nodes -- the reference's per-local-slot nodal
    // vectors (exDyna3D.cpp:523-634), each entry written by the one element
    // that holds the node in slot k (or has row k at the node); 0: elements,
    // gathered through ell / csr by the node pass
    int32_t slot_major;
    int32_t bt9;               // FP64: bt holds 9 numbers per element (else 24)
    int32_t pad;
};

// Entry e of a component array: its rows start at tile_row(E, p, e), `stride`
// entries apart (tile_stride), with the element at e & 31.
template <typename T>
__host__ __device__ inline T* tile_row(const ElemArrays& E, T* p, int64_t e) {
    if (E.tile_bytes) {
        using B = const char;
        return const_cast<T*>(reinterpret_cast<const T*>(reinterpret_cast<B*>(p) + (e >> 5) * E.tile_bytes));
    }
    return p + (e & ~int64_t(31));
}
__host__ __device__ inline int64_t tile_stride(const ElemArrays& E) { return E.tile_bytes ? 32 : E.ne_pad; }

// Elements per patch of the mixed patch assembly: one staged tile.
constexpr int kPatchElems = 64;

// The tables of the patch assembly (mixed precision), kept apart from the
// element and node arrays so that kernels of the slot assembly see the same
// argument layout either way; all null for an instance on the slot
// assembly.  Elements are stored in patches of kPatchElems consecutive
// elements.  The element pass sums a patch's element forces per patch node
// in shared memory and writes one partial per (patch, node): patch p's
// nodes are the partial entries pf_off[p] .. pf_off[p + 1] - 1, entry q's
// incidences are pinc[pinc_off[q] .. pinc_off[q + 1]) as (element in patch
// << 3 | slot), in slot order, and its partial goes to pf[c * pf_pad + q].
// Node n's force is the sum of its partials nent[nptr[n] .. nptr[n + 1]),
// in patch order.  iperm (also without patches; null: the same) maps an element
// of the caller's numbering to its stored position.
struct PatchArrays {
    const uint32_t* pf_off;
    const uint32_t* pinc_off;
    const uint16_t* pinc;
    float* pf;
    int64_t pf_pad;
    const uint32_t* nptr;
    const uint32_t* nent;
    const int32_t* iperm;
};

struct NodeArrays {
    int64_t nn, nn_pad;
    double* x;
    double* u;
    void* v;                   // double (FP64) or float (mixed)
    const double* inv_mass;
    const uint8_t* bc;
    const double* bcv;
    const uint32_t* ell;
    const int64_t* csr_ptr;    // non-null: use the general lists
    const uint32_t* csr_ent;   // (e << 3) | slot
    const uint8_t* merge;      // with ElemArrays::rows: bit r set where row r holds the same slot as row r - 1
    double* rf;                // reactions, [3][nn_pad]
    int32_t rec;               // 1: x, u, v in records (head of this file), 0: rows
    int32_t pad;
};

// Force hand-off of slot k, entry i (a node or an element; `np` entries per
// row): (fx, fy) and fz.
template <typename T>
__host__ __device__ inline T* force_xy(T* fe, int64_t np, int k, int64_t i) {
    return fe + 2 * (k * np + i);
}
template <typename T>
__host__ __device__ inline T* force_z(T* fe, int64_t np, int k, int64_t i) {
    return fe + (16 + k) * np + i;
}

// Partial sums written by each block of a pass, folded in fixed block order.
struct Partials {
    double* elem;              // [3][n_elem_blocks]
    double* node;              // [2][n_node_blocks]
    int32_t n_elem_blocks, n_node_blocks;
};

// The node pass's view of one instance: node arrays, slot-major forces,
// gravity and the control block.  `grouped` is 1 when the forces are
// slot-major and the rows tile-aligned, so W consecutive nodes can be read
// and written as vectors, and 2 for the same under the patch assembly.  In
// a batch, two 128-byte lines per slot; the second is read only under the
// patch assembly.
struct alignas(128) NodeView {
    const void* fe;
    void* v;                   // double (FP64) or float (mixed)
    double* u;
    double* x;
    const double* inv_mass;
    const uint8_t* bc;
    const uint8_t* merge;      // NodeArrays::merge
    double* rf;
    Ctl* ctl;
    int64_t nn, np;
    double gravity_value, gravity_dir[3];
    int32_t gravity_on;
    int32_t grouped;
    // patch assembly (pf non-null): node n's force is the sum of
    // pf[c * pf_pad + nent[i]] over i in [nptr[n], nptr[n + 1])
    const float* pf;
    const uint32_t* nptr;
    const uint32_t* nent;
    int64_t pf_pad;
};
static_assert(sizeof(NodeView) == 256, "two lines per slot");

__host__ __device__ inline NodeView node_view(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl,
                                              const PatchArrays* pa = nullptr) {
    NodeView v{};
    v.fe = E.fe;
    v.v = N.v;
    v.u = N.u;
    v.x = N.x;
    v.inv_mass = N.inv_mass;
    v.bc = N.bc;
    v.merge = N.merge;
    v.rf = N.rf;
    v.ctl = ctl;
    v.nn = N.nn;
    v.np = N.nn_pad;
    v.gravity_value = M.gravity_value;
    for (int c = 0; c < 3; ++c) v.gravity_dir[c] = M.gravity_dir[c];
    v.gravity_on = M.gravity_on;
    const bool patch = pa && pa->pf;
    v.grouped = (E.slot_major && E.tile_bytes) ? (patch ? 2 : 1) : 0;
    if (patch) {
        v.pf = pa->pf;
        v.nptr = pa->nptr;
        v.nent = pa->nent;
        v.pf_pad = pa->pf_pad;
    }
    return v;
}

// ---- batched instances ------------------------------------------------------
// Independent solver instances advanced together: each warp-sized tile (32
// elements or 32 nodes) belongs to one instance, so instance parameters,
// clock and reductions are warp-uniform.
constexpr int kTile = 32;

// The scalars of an instance's node pass in the current cycle (stable dt,
// previous dt, gravity amplitude), computed once per instance.
struct alignas(16) NodeParam {
    double dt_i, dt_i_1, amp;
    int32_t live, pad;
};

// The scalars of an instance's element pass in the current cycle (dt_i_1,
// and whether it runs), written per slot at the start of the cycle and
// bulk-copied into the stage of each of its element tiles.
struct StageHdr {
    double dt1;
    int32_t live, pad;
};

// Where the batch element passes copy an element tile from.  A tile's record
// travels with the stage of the tile two visits earlier, so the warp that copies
// a tile reads its record from shared memory.
struct alignas(16) ETileSrc {
    const void* tile;
    int32_t bytes;    // of the tiles the pass takes at once
    int32_t slot, base;
    int32_t pad[3];
};
static_assert(sizeof(ETileSrc) == 32, "tile records are bulk-copied");

// Written into each stage by the thread that fills it: the tile's instance
// slot and first element.
struct TileInfo {
    int32_t slot, base, pad0, pad1;
};

struct alignas(16) InstanceDesc {
    ElemArrays E;
    NodeArrays N;
    Material M;
    Ctl* ctl;
    int32_t e_tile0, e_ntiles;   // range in the element-tile list
    int32_t n_tile0, n_ntiles;   // range in the node-tile list
    int32_t active;
    int32_t patch;               // 1: the patch assembly, tables in pa
    PatchArrays pa;
};

struct BatchTables {
    const InstanceDesc* desc;    // [slots]
    Ctl* ctl;                    // [slots] control blocks (desc[s].ctl is ctl + s)
    const int32_t* etile_inst;   // [etiles] instance slot of each element tile
    const int32_t* etile_base;   // first element of the tile within its instance
    const int32_t* ntile_inst;   // [ntiles]
    const int32_t* ntile_base;
    const int32_t* counts;       // [0] element tiles, [1] node tiles, [2] slots in use
    // per-tile energy terms: work done since the last fold (internal,
    // hourglass, viscous; external) and the latest kinetic energy
    double* etile_part;          // [etiles][etile / 32][3] internal / hourglass / viscous work per tile warp
    double* ntile_part;          // [ntiles][2] kinetic energy / external work per tile
    int32_t* exact_count;        // instances whose current cycle needs the edge prepass
    int32_t* prepass_done;       // blocks of the edge prepass that have finished
    int32_t* elem_done;          // blocks of the element pass that have finished
    NodeParam* nparam;           // [slots] this cycle's node-pass scalars
    StageHdr* sparam;            // [slots] this cycle's element-pass scalars
    const NodeView* nview;       // [slots]
    const ETileSrc* etile_src;   // [etiles] copy sources of each element tile
    int32_t etile, ntile;        // elements / nodes per tile
    int32_t tile_room;           // bytes the stages of the element pass have for a tile
    int32_t pad;
};
static_assert(sizeof(InstanceDesc) % 16 == 0, "instance descriptors are bulk-copied");
// behind the tile in a stage of the batched element passes: the descriptor, then
constexpr uint32_t kBatchHdrOff = sizeof(InstanceDesc);
constexpr uint32_t kBatchInfoOff = kBatchHdrOff + sizeof(StageHdr);
constexpr uint32_t kBatchNextOff = kBatchInfoOff + sizeof(TileInfo);
constexpr uint32_t kBatchTailBytes = (kBatchNextOff + sizeof(ETileSrc) + 127) / 128 * 128;
static_assert(sizeof(StageHdr) == 16 && sizeof(TileInfo) == 16, "16-byte copies");

// Amplitude factor of gravity in a cycle at `time` with step dt, as
// exDyna3D::deal_amp computes it (exDyna3D.cpp:1222-1278), behaviour kept as
// is: the scan stops at the first segment that ends before `time` (factor
// 1); a cycle inside one segment takes the segment's value at mid-cycle; a
// cycle that crosses segment ends takes the mean of the curve over the cycle,
// where the partial last segment's intercept uses the first segment's slope
// (:1257) and time past the last point counts with value 1.  n < 2: 1.
__host__ __device__ inline double gravity_amplitude(const double* amp, int n, double time, double dt) {
    double y = 1.0;
    for (int i = 0; i + 1 < n; ++i) {
        const double x1 = amp[2 * i], y1 = amp[2 * i + 1];
        const double x2 = amp[2 * i + 2], y2 = amp[2 * i + 3];
        if (time > x2) break;
        const double m = (y2 - y1) / (x2 - x1);
        const double c = y1 - m * x1;
        const double x = time + dt / 2.0;
        if ((x + dt / 2.0) < x2) {
            y = m * x + c;
            break;
        }
        const double dt1 = x2 - time;
        const double xm = time + dt1 / 2.0;
        const double ym = m * xm + c;
        const double a1 = ym * dt1;
        double a2 = 0.0;
        for (int j = 2; j + i < n; ++j) {
            const double xj = amp[2 * (i + j)], yj = amp[2 * (i + j) + 1];
            const double xp = amp[2 * (i + j - 1)], yp = amp[2 * (i + j - 1) + 1];
            if ((x + dt / 2.0) > xj) {
                a2 += (xj - xp) * (yj + yp) / 2.0;
            } else {
                const double mj = (yj - yp) / (xj - xp);
                const double cj = yp - m * xp;
                const double yend = mj * (x + dt / 2.0) + cj;
                a2 += (x + dt / 2.0 - xp) * (yp + yend) / 2.0;
                break;
            }
        }
        const double x_end = amp[2 * (n - 1)];
        if (x + dt / 2.0 > x_end) a2 += (x + dt / 2.0 - x_end) * 1.0;
        y = (a1 + a2) / dt;
        break;
    }
    return y;
}

// ---- mixed-precision velocities ---------------------------------------------
// The mixed stepper keeps each velocity component as a float `hi` (what the
// element pass reads) and a 16-bit residual `lo` in units of 2^-16 of hi's
// spacing: v = hi + lo * ulp(hi) / 2^16, about 40 significant bits.  The node
// pass updates v in FP64 and splits it again, so the velocity integration
// does not drop FP32 rounding every cycle.

// The mixed stepper's element pass forms F from the current coordinates and
// never reads the displacement, so it keeps the reference position
// xr = x - u in the u rows instead of u, and the node pass updates x alone:
// u = x - xr is formed where the state is read (ensc_download, snapshots),
// and an upload of x or u sets xr = x - u.  Both are FP64: u = x - xr is
// within a rounding of x's magnitude of the separately accumulated u.

// ulp(hi) / 2^16 and its inverse (normal or zero hi; hi's exponent field e
// gives ulp(hi) = 2^(e - 150), with e = 1 for zero and subnormals)
__host__ __device__ inline double vlo_unit(float hi) {
    uint32_t b;
    memcpy(&b, &hi, sizeof b);
    int e = static_cast<int>((b >> 23) & 0xFFu);
    if (e == 0) e = 1;
    const uint64_t d = static_cast<uint64_t>(e - 166 + 1023) << 52;
    double r;
    memcpy(&r, &d, sizeof r);
    return r;
}
__host__ __device__ inline double vlo_inv_unit(float hi) {
    uint32_t b;
    memcpy(&b, &hi, sizeof b);
    int e = static_cast<int>((b >> 23) & 0xFFu);
    if (e == 0) e = 1;
    const uint64_t d = static_cast<uint64_t>(166 - e + 1023) << 52;
    double r;
    memcpy(&r, &d, sizeof r);
    return r;
}
__host__ __device__ inline double v_join(float hi, int16_t lo) {
    return static_cast<double>(hi) + static_cast<double>(lo) * vlo_unit(hi);
}
__host__ __device__ inline void v_split(double v, float& hi, int16_t& lo) {
    hi = static_cast<float>(v);
    double q = rint((v - static_cast<double>(hi)) * vlo_inv_unit(hi));
    if (!(q >= -32768.0 && q <= 32767.0)) q = q > 0.0 ? 32767.0 : -32768.0;  // |q| <= 2^15; NaN -> bound
    lo = static_cast<int16_t>(q);
}
// the residual rows of a mixed velocity array
__host__ __device__ inline int16_t* v_lo_rows(void* v, int64_t nn_pad) {
    return reinterpret_cast<int16_t*>(static_cast<float*>(v) + nn_pad);
}

// One entry of the node state in either layout (FP64 displacement; the mixed
// u rows are plain).
__host__ __device__ inline double* node_x(const NodeArrays& N, int c, int64_t n) {
    return N.rec ? N.x + 4 * n + c : N.x + c * N.nn_pad + n;
}
__host__ __device__ inline double* node_u64(const NodeArrays& N, int c, int64_t n) {
    if (!N.rec) return N.u + c * N.nn_pad + n;
    return c == 0 ? N.x + 4 * n + 3 : N.u + 4 * n + (c - 1);
}
__host__ __device__ inline double* node_v64(const NodeArrays& N, int c, int64_t n) {
    double* v = static_cast<double*>(N.v);
    if (!N.rec) return v + c * N.nn_pad + n;
    return c < 2 ? N.u + 4 * n + 2 + c : v + n;
}
__host__ __device__ inline float* node_vf(const NodeArrays& N, int c, int64_t n) {
    return c < 2 ? reinterpret_cast<float*>(N.x + 4 * n + 3) + c : static_cast<float*>(N.v) + n;
}

// A node record: 32 bytes in one load or store.  The load is volatile, as a
// resident run's records change between its cycles.
__device__ __forceinline__ void ld_rec(const double* p, double (&o)[4]) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3])
                 : "l"(p));
}
__device__ __forceinline__ void st_rec(double* p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}
// the two floats of a mixed record's fourth word
__device__ __forceinline__ float rec_vx(double w) { return __int_as_float(__double2loint(w)); }
__device__ __forceinline__ float rec_vy(double w) { return __int_as_float(__double2hiint(w)); }
__device__ __forceinline__ double rec_vxy(float vx, float vy) {
    return __hiloint2double(__float_as_int(vy), __float_as_int(vx));
}

// Vector access to W consecutive entries of a padded SoA row (rows start
// 256-byte aligned, the row stride is a multiple of 32 entries and the first
// index a multiple of W): 16-byte chunks, or one 8-byte chunk when the W
// entries take 8 bytes.
template <int W, typename T>
__device__ __forceinline__ void ld_row(const T* p, T (&o)[W]) {
    constexpr int kBytes = W * static_cast<int>(sizeof(T));
    static_assert(kBytes % 16 == 0 || kBytes == 8 || kBytes == 4 || W == 1, "16-byte chunks or one smaller chunk");
    if constexpr (W == 1) {
        o[0] = *p;
    } else if constexpr (kBytes == 4) {
        const uint32_t q = *reinterpret_cast<const uint32_t*>(p);
        memcpy(o, &q, 4);
    } else if constexpr (kBytes == 8) {
        const uint2 q = *reinterpret_cast<const uint2*>(p);
        memcpy(o, &q, 8);
    } else {
#pragma unroll
        for (int i = 0; i < kBytes / 16; ++i) {
            const uint4 q = reinterpret_cast<const uint4*>(p)[i];
            memcpy(reinterpret_cast<char*>(o) + 16 * i, &q, 16);
        }
    }
}
template <int W, typename T>
__device__ __forceinline__ void st_row(T* p, const T (&v)[W]) {
    constexpr int kBytes = W * static_cast<int>(sizeof(T));
    static_assert(kBytes % 16 == 0 || kBytes == 8 || kBytes == 4 || W == 1, "16-byte chunks or one smaller chunk");
    if constexpr (W == 1) {
        *p = v[0];
    } else if constexpr (kBytes == 4) {
        uint32_t q;
        memcpy(&q, v, 4);
        *reinterpret_cast<uint32_t*>(p) = q;
    } else if constexpr (kBytes == 8) {
        uint2 q;
        memcpy(&q, v, 8);
        *reinterpret_cast<uint2*>(p) = q;
    } else {
#pragma unroll
        for (int i = 0; i < kBytes / 16; ++i) {
            uint4 q;
            memcpy(&q, reinterpret_cast<const char*>(v) + 16 * i, 16);
            reinterpret_cast<uint4*>(p)[i] = q;
        }
    }
}
// W (1, 2 or 4) consecutive bytes as one word, byte j of node j in bits 8j..8j+7.
template <int W>
__device__ __forceinline__ uint32_t ld_bytes(const uint8_t* p) {
    static_assert(W == 1 || W == 2 || W == 4, "1, 2 or 4 bytes");
    if (W == 1) return *p;
    if (W == 4) return *reinterpret_cast<const uint32_t*>(p);
    return *reinterpret_cast<const uint16_t*>(p);
}

// A NodeView of a batch table through the non-coherent (L1-cached) path:
// the table does not change while a pass runs.
__device__ __forceinline__ NodeView ld_view(const NodeView* p) {
    constexpr int kW = sizeof(NodeView) / sizeof(uint4);
    uint4 w[kW];
#pragma unroll
    for (int i = 0; i < kW; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
    NodeView v;
    memcpy(&v, w, sizeof(v));
    return v;
}
__device__ __forceinline__ NodeParam ld_param(const NodeParam* p) {
    uint4 w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
    NodeParam v;
    memcpy(&v, w, sizeof(v));
    return v;
}
// ---- programmatic launches (launch_cycle_kernel) ----
// A kernel launched while the one before it still runs waits here until that
// one has completed and its writes are visible.  Only then may the next be
// launched, so that what the kernel before the last one wrote can be read
// ahead of the wait.
__device__ __forceinline__ void cycle_kernel_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Read-only input loads: through the non-coherent path from global memory,
// plain loads from a shared-memory stage.
template <bool SMEM, typename T>
__device__ __forceinline__ T ldin(const T* p) {
    if constexpr (SMEM) return *p;
    else return __ldg(p);
}

// The node pass's scalars of one batch slot: this cycle's stable dt
// (update_minVertex_perMaterial_and_dt, exDyna3D.cpp:673-679, as the
// single-instance node pass computes it), the previous dt and the gravity
// amplitude; also the control-block updates that pass makes.  Run by the
// last block of the batched element pass, after every block's minima: the
// edge minimum is read through L2.
__device__ inline void node_params_slot(const BatchTables& T, int slot) {
    const InstanceDesc& d = T.desc[slot];
    Ctl* ctl = T.ctl + slot;
    NodeParam p{0.0, 0.0, 1.0, 0, 0};
    // all that it may need at once, not load after branch
    const int active = d.active, gravity = d.M.gravity_on && d.M.amp_n > 0;
    const int done = ctl->done, dt_final = ctl->dt_final;
    const double len = __longlong_as_double(static_cast<long long>(__ldcg(&ctl->len_min)));
    const double wos = ctl->wos, dts = ctl->dts_cur, factor = ctl->factor, time = ctl->time, fixed = ctl->dt_i;
    const double dt_i_1 = ctl->dt_i_1;
    const long long cycles = ctl->cycles_done;
    if (active && !done) {
        double dt_i = fixed;
        if (!dt_final) {
            double dd = len / wos;
            dd = dd < dts ? dd : dts;
            dt_i = dd * factor;
        }
        if (!(dt_i > 0.0) || !isfinite(dt_i)) atomicOr(&ctl->status, ST_BAD_DT);
        if (!dt_final) ctl->dt_i = dt_i;
        ctl->cycles_done = cycles + 1;
        ctl->energy_pending = 1;
        p.dt_i = dt_i;
        p.dt_i_1 = dt_i_1;
        p.amp = gravity ? gravity_amplitude(d.M.amp, d.M.amp_n, time, dt_i) : 1.0;
        p.live = 1;
    }
    T.nparam[slot] = p;
}

// Called by every block of a batched element pass after its last tile: the
// last block to finish fills the node pass's scalars of all slots.
__device__ inline void element_pass_done(const BatchTables& T) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(T.elem_done, 1) == static_cast<int>(gridDim.x) - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int slot = threadIdx.x; slot < T.counts[2]; slot += blockDim.x) node_params_slot(T, slot);
    if (threadIdx.x == 0) *T.elem_done = 0;
}

// Positive doubles order like their bit patterns; min-reductions over
// element dt / edge lengths use integer atomicMin on the bits, which is
// exact and independent of scheduling.
__device__ __forceinline__ unsigned long long ord_bits(double d) {
    return static_cast<unsigned long long>(__double_as_longlong(d));
}
__device__ __forceinline__ double bits_ord(unsigned long long b) {
    return __longlong_as_double(static_cast<long long>(b));
}
constexpr unsigned long long kInfBits = 0x7FF0000000000000ull;

}  // namespace ensc
