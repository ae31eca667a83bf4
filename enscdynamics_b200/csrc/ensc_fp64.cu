// Plain FP64 stepper kernels.  Compiled with -fmad=false: every product and
// sum below is rounded separately, in the order written, which is the order
// the reference evaluates it (cited per block), so results match the
// reference CPU stepper to round-off and the CPU restatement bit-for-bit.
//
// One cycle (exDyna3D::run loop body, Explicit3D/source/exDyna3D.cpp:86-100)
// is the kernel sequence
//   begin  -> [edge_prepass -> begin_exact] -> element -> node
// launched inside a CUDA graph, or the phases of a resident run
// (ensc_run.cuh); see ensc_capi.cu for the orchestration.
#include "ensc_device.cuh"
#include "ensc_kernels.h"
#include "ensc_run.cuh"
#include "ensc_stage.cuh"

#include <algorithm>
#include <cfloat>
#include <type_traits>

namespace ensc {
namespace {

__device__ __forceinline__ double det3(const double m[3][3]) {
    // Eigen 3.4 bruteforce_det3_helper form (Eigen/src/LU/Determinant.h),
    // as used by all_F[e].determinant() (exDyna3D.cpp:869).
    const double h0 = m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1]);
    const double h1 = m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0]);
    const double h2 = m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
    return (h0 - h1) + h2;
}

__device__ __forceinline__ double cof3(const double m[3][3], int i, int j) {
    const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
    return m[i1][j1] * m[i2][j2] - m[i1][j2] * m[i2][j1];
}

__device__ __forceinline__ void inv3(const double m[3][3], double r[3][3]) {
    // Eigen 3.4 compute_inverse<...,3> (Eigen/src/LU/InverseImpl.h), as used
    // by all_F[e].inverse() (exDyna3D.cpp:874).
    const double c0 = cof3(m, 0, 0), c1 = cof3(m, 1, 0), c2 = cof3(m, 2, 0);
    const double det = (c0 * m[0][0] + c1 * m[1][0]) + c2 * m[2][0];
    const double invdet = 1.0 / det;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) r[i][j] = cof3(m, j, i) * invdet;
}

template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const T w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w < v ? w : v;
    }
    return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Fixed-shape block reduction (warp butterflies, then warp 0 over the
// warp results): deterministic for a given block size.
// Block sum of NV values into out_slots[i * stride + slot]; values whose bit
// is set in ACC are added to the slot (it accumulates over cycles, one writer
// per slot and pass), the others stored.
template <int NT, int NV, unsigned ACC = 0u>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* out_slots, int stride, int slot) {
    __shared__ double red[NV][NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const double s = warp_sum(v[i]);
        if (lane == 0) red[i][wid] = s;
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double s = lane < NT / 32 ? red[i][lane] : 0.0;
            s = warp_sum(s);
            if (lane == 0) {
                double* o = out_slots + i * stride + slot;
                if ((ACC >> i) & 1u) atomicAdd(o, s);
                else *o = s;
            }
        }
    }
    __syncthreads();
}

template <int NT>
__device__ __forceinline__ void block_min2(double a, double b, unsigned long long* ga, unsigned long long* gb) {
    __shared__ unsigned long long ra[NT / 32], rb[NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long x = warp_min(ord_bits(a)), y = warp_min(ord_bits(b));
    if (lane == 0) {
        ra[wid] = x;
        rb[wid] = y;
    }
    __syncthreads();
    if (wid == 0) {
        x = lane < NT / 32 ? ra[lane] : kInfBits;
        y = lane < NT / 32 ? rb[lane] : kInfBits;
        x = warp_min(x);
        y = warp_min(y);
        if (lane == 0) {
            if (ga) atomicMin(ga, x);
            if (gb) atomicMin(gb, y);
        }
    }
    __syncthreads();
}

// Where one element's inputs are read from: rows of `stride` entries with the
// element at `i`, in the instance's tiles or rows in global memory or in a tile
// in shared memory.
struct Fp64Src {
    const uint32_t* conn;   // [8] rows
    const double* bt;       // [9] or [24] rows
    const double* vol0;
    const double* cb;       // cbrt(V0)
    const double* cb2;      // cbrt(V0^2)
    const double* sig;      // [6] rows
    const double* qia;      // [12] rows
    const double* eps;
    int64_t stride, i;
};

// TILED: the instance's arrays are in tiles, else plain rows (ElemArrays).
template <bool TILED>
__device__ __forceinline__ Fp64Src fp64_src_global(const ElemArrays& E, int64_t e) {
    if constexpr (!TILED)
        return Fp64Src{E.conn,
                       static_cast<const double*>(E.bt),
                       E.vol0,
                       static_cast<const double*>(E.cbrt_v0),
                       E.cbrt_v0sq,
                       static_cast<const double*>(E.sigma),
                       static_cast<const double*>(E.qia),
                       static_cast<const double*>(E.eps_p),
                       E.ne_pad,
                       e};
    return Fp64Src{tile_row(E, E.conn, e),
                   tile_row(E, static_cast<const double*>(E.bt), e),
                   tile_row(E, E.vol0, e),
                   tile_row(E, static_cast<const double*>(E.cbrt_v0), e),
                   tile_row(E, E.cbrt_v0sq, e),
                   tile_row(E, static_cast<const double*>(E.sigma), e),
                   tile_row(E, static_cast<const double*>(E.qia), e),
                   tile_row(E, static_cast<const double*>(E.eps_p), e),
                   32,
                   e & 31};
}

// Where one element's evolving rows are written: the instance's own arrays, or
// the shared-memory tile that a resident run keeps them in.
struct Fp64Out {
    double* sig;            // [6] rows
    double* qia;            // [12] rows
    double* eps;
    int64_t stride, i;
};

template <bool TILED>
__device__ __forceinline__ Fp64Out fp64_out_global(const ElemArrays& E, int64_t e) {
    if constexpr (!TILED)
        return Fp64Out{static_cast<double*>(E.sigma), static_cast<double*>(E.qia), static_cast<double*>(E.eps_p),
                       E.ne_pad, e};
    return Fp64Out{tile_row(E, static_cast<double*>(E.sigma), e), tile_row(E, static_cast<double*>(E.qia), e),
                   tile_row(E, static_cast<double*>(E.eps_p), e), 32, e & 31};
}

// A tile of layout L (Fp64Tile9 / Fp64Tile24) in memory: row pointers of the
// element at `lane`.
template <typename L>
__device__ __forceinline__ Fp64Src fp64_src_tile(const unsigned char* t, int lane) {
    return Fp64Src{reinterpret_cast<const uint32_t*>(t),
                   reinterpret_cast<const double*>(t + L::kBt),
                   reinterpret_cast<const double*>(t + L::kVol0),
                   reinterpret_cast<const double*>(t + L::kCb),
                   reinterpret_cast<const double*>(t + L::kCb + L::kRow),
                   reinterpret_cast<const double*>(t + L::kSig),
                   reinterpret_cast<const double*>(t + L::kQia),
                   reinterpret_cast<const double*>(t + L::kEps),
                   32,
                   lane};
}
template <typename L>
__device__ __forceinline__ Fp64Out fp64_out_tile(unsigned char* t, int lane) {
    return Fp64Out{reinterpret_cast<double*>(t + L::kSig), reinterpret_cast<double*>(t + L::kQia),
                   reinterpret_cast<double*>(t + L::kEps), 32, lane};
}

// The four Gamma-signed sums of 8 values, each left to right from node 0 as
// the oracle adds them; rows that agree up to sign so far share their partial
// sum (rounding is symmetric in sign), 24 additions instead of 28.
__device__ __forceinline__ void gamma_sums(const double (&v)[8], double (&t)[4]) {
    const double d = v[0] - v[1], s = v[0] + v[1], q = (d + v[2]) - v[3];
    t[0] = (((q + v[4]) - v[5]) + v[6]) - v[7];
    t[1] = (((((v[2] - s) + v[3]) + v[4]) + v[5]) - v[6]) - v[7];
    t[2] = (((((v[2] - d) - v[3]) + v[4]) - v[5]) - v[6]) + v[7];
    t[3] = (((v[4] - q) - v[5]) + v[6]) - v[7];
}

// B0^T rows of an element.  9 numbers p = J^-1 / 8: row a is
// (+-p0 +- p1) +- p2 with the corner signs of node a, and opposite corners have
// opposite rows, so 4 rows of 3 carry all 8.  24 numbers: as stored.
template <bool BT9, bool SMEM>
struct B0Rows {
    double r[4][3];  // BT9: nodes 6, 1, 2, 5
    __device__ __forceinline__ void load(const Fp64Src& S) {
        const double* b = S.bt + S.i;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double p0 = ldin<SMEM>(b + (3 * c) * S.stride), p1 = ldin<SMEM>(b + (3 * c + 1) * S.stride),
                         p2 = ldin<SMEM>(b + (3 * c + 2) * S.stride);
            const double u = p0 + p1, w = p0 - p1;
            r[0][c] = u + p2;
            r[1][c] = w - p2;
            r[2][c] = u - p2;
            r[3][c] = w + p2;
        }
    }
    // row of node j: minus(j) ? -r[index(j)] : r[index(j)]
    __device__ static constexpr int index(int j) {
        constexpr int k[8] = {0, 1, 2, 3, 2, 3, 0, 1};
        return k[j];
    }
    __device__ static constexpr bool minus(int j) { return j == 0 || j == 3 || j == 4 || j == 7; }
    __device__ __forceinline__ double at(int j, int c) const { return minus(j) ? -r[index(j)][c] : r[index(j)][c]; }
    // 24 numbers: row j as stored
    __device__ __forceinline__ void row(const Fp64Src& S, int j, double (&bb)[3]) const {
#pragma unroll
        for (int c = 0; c < 3; ++c) bb[c] = ldin<SMEM>(S.bt + (3 * j + c) * S.stride + S.i);
    }
};

// Gamma row k, node j is +1 (exDyna3D.cpp:1003-1008).
__device__ __forceinline__ constexpr bool gamma_plus(int k, int j) {
    constexpr unsigned kMask = 0x55u | (0x3Cu << 8) | (0x96u << 16) | (0x5Au << 24);
    return (kMask >> (8 * k + j)) & 1u;
}

// One element of the FP64 element pass (the kernel comment below has the
// reference mapping), shared by the single-instance, batched and resident-run
// kernels; inputs come from S, the evolving rows go to O and the forces to the
// instance's force array at element e.  Node rows are read with plain loads: a
// resident run rewrites them between its cycles.  SMEM: S's rows are in shared
// memory.  BT9: its bt rows are the 9-number form.  REC: node records (three
// loads per node; a record's last numbers are read when F and the velocity
// gradient need them), else plain rows.  PF: the second record and vz of each
// node are prefetched into L1 once the connectivity is known.
template <bool PLASTIC, bool INIT, bool BT9, bool REC, bool SMEM = false, bool PF = false>
__device__ __forceinline__ void element_body(const ElemArrays& E, const NodeArrays& N, const Material& M,
                                             const Fp64Src& S, const Fp64Out& O, const double dt1, const int64_t e,
                                             double& dts, double& len, double& e_int, double& e_hg, double& e_vis,
                                             int32_t& bad) {
    const int64_t ss = S.stride, si = S.i, os = O.stride, oi = O.i;
    const int64_t np = N.nn_pad;
    const double* X = N.x;
    const double* U = N.u;
    const double* V = static_cast<const double*>(N.v);
    const double G = M.G, lam = M.lambda;

    uint32_t n[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) n[k] = ldin<SMEM>(S.conn + k * ss + si);
    if (REC && E.rows) prefetch_l1(E.rows + e);  // read with the forces
    if constexpr (REC && PF) {
#pragma unroll
        for (int k = 0; k < 8; ++k) prefetch_l1(U + 4 * static_cast<int64_t>(n[k]));
#pragma unroll
        for (int k = 0; k < 8; ++k) prefetch_l1(V + n[k]);
    }
    // current coordinates: hourglass projections TAU x and the minimum edge
    // (min_ele_edge :1173-1220)
    double TX[4][3], ux[8];
    {
        double xyz[8][3];
        if constexpr (REC) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                double q[4];
                ld_rec(X + 4 * static_cast<int64_t>(n[k]), q);
#pragma unroll
                for (int c = 0; c < 3; ++c) xyz[k][c] = q[c];
                ux[k] = q[3];
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int c = 0; c < 3; ++c) xyz[k][c] = X[c * np + n[k]];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double x[8], t[4];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = xyz[k][c];
            gamma_sums(x, t);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) TX[kk][c] = t[kk];
        }
        len = sqrt(min_edge_sq(xyz));
    }
    // the second records: uy, uz, vx, vy
    double q1[8][4];
    if constexpr (REC) {
#pragma unroll
        for (int k = 0; k < 8; ++k) ld_rec(U + 4 * static_cast<int64_t>(n[k]), q1[k]);
    }
    auto u_at = [&](int r, int k) -> double {
        if constexpr (REC) return r == 0 ? ux[k] : q1[k][r - 1];
        else return U[r * np + n[k]];
    };
    auto v_at = [&](int r, int k) -> double {
        if constexpr (REC) return r < 2 ? q1[k][2 + r] : V[n[k]];
        else return V[r * np + n[k]];
    };
    // F = I + u_e B0^T (:862-865); with B0 in its 9-number form one component
    // at a time, else node by node (24 numbers would stay in registers)
    B0Rows<BT9, SMEM> B;
    double F[3][3];
    if constexpr (BT9) {
        B.load(S);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double u[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) u[k] = u_at(r, k);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double t = 0.0;
#pragma unroll
                for (int k = 0; k < 8; ++k) t = __fma_rn(u[k], B.at(k, c), t);
                F[r][c] = t;
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) F[i / 3][i % 3] = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            double bb[3];
            B.row(S, k, bb);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const double u = u_at(r, k);
#pragma unroll
                for (int c = 0; c < 3; ++c) F[r][c] = __fma_rn(u, bb[c], F[r][c]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) F[r][r] = 1.0 + F[r][r];
    const double J = det3(F);
    double Fi[3][3];
    inv3(F, Fi);
    if (!(J > 0.0)) bad |= ST_INVERTED;
    // L0 = v_e B0^T, VT = v_e Gamma^T (signed sums), NX2 (:1024)
    double L0[3][3], VT[3][4], nx2 = 0.0;
    if constexpr (BT9) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = v_at(r, j);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double l = 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j) l = __fma_rn(v[j], B.at(j, c), l);
                L0[r][c] = l;
            }
            gamma_sums(v, VT[r]);
        }
        double sq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            sq[j] = __fma_rn(B.r[j][2], B.r[j][2], __fma_rn(B.r[j][1], B.r[j][1], B.r[j][0] * B.r[j][0]));
#pragma unroll
        for (int j = 0; j < 8; ++j) nx2 = nx2 + sq[B.index(j)];
    } else {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
            for (int c = 0; c < 3; ++c) L0[r][c] = 0.0;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) VT[r][kk] = 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            double bb[3];
            B.row(S, j, bb);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const double v = v_at(r, j);
#pragma unroll
                for (int c = 0; c < 3; ++c) L0[r][c] = __fma_rn(v, bb[c], L0[r][c]);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) VT[r][kk] = gamma_plus(kk, j) ? VT[r][kk] + v : VT[r][kk] - v;
            }
            nx2 = nx2 + __fma_rn(bb[2], bb[2], __fma_rn(bb[1], bb[1], bb[0] * bb[0]));
        }
    }
    // L = L0 F^-1 (= v_e b^T, :928); HIA = VT - L0 TX^T (= v_e ATAU^T, :1020-1021)
    double L[3][3], HIA[3][4];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
            L[r][c] = __fma_rn(L0[r][2], Fi[2][c], __fma_rn(L0[r][1], Fi[1][c], L0[r][0] * Fi[0][c]));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
            HIA[r][kk] = VT[r][kk] - __fma_rn(L0[r][2], TX[kk][2], __fma_rn(L0[r][1], TX[kk][1], L0[r][0] * TX[kk][0]));
    }
    const double vr = (L[0][0] + L[1][1]) + L[2][2];
    // Jaumann stress update (:930-973)
    double eps[6];
    eps[0] = L[0][0] * dt1;
    eps[1] = L[1][1] * dt1;
    eps[2] = L[2][2] * dt1;
    eps[3] = (L[0][1] + L[1][0]) / 2.0 * dt1;
    eps[4] = (L[0][2] + L[2][0]) / 2.0 * dt1;
    eps[5] = (L[1][2] + L[2][1]) / 2.0 * dt1;
    const double w0 = (L[0][1] - L[1][0]) / 2.0;
    const double w1 = (L[0][2] - L[2][0]) / 2.0;
    const double w2 = (L[1][2] - L[2][1]) / 2.0;
    const double tr = (eps[0] + eps[1]) + eps[2];
    double s[6], so[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) so[i] = S.sig[i * ss + si];
    double inc[6];
    inc[0] = (lam * tr + 2.0 * G * eps[0]) + 2.0 * so[3] * w0 * dt1 + 2.0 * so[4] * w1 * dt1;
    inc[1] = (lam * tr + 2.0 * G * eps[1]) - 2.0 * so[3] * w0 * dt1 + 2.0 * so[5] * w2 * dt1;
    inc[2] = (lam * tr + 2.0 * G * eps[2]) - 2.0 * so[4] * w1 * dt1 - 2.0 * so[5] * w2 * dt1;
    inc[3] = (2.0 * G * eps[3]) + (so[1] - so[0]) * w0 * dt1 + so[5] * w1 * dt1;
    inc[4] = (2.0 * G * eps[4]) + (so[2] - so[0]) * w1 * dt1 + so[5] * w0 * dt1;
    inc[5] = (2.0 * G * eps[5]) + (so[2] - so[1]) * w2 * dt1 + so[3] * w1 * dt1 - so[4] * w0 * dt1;
#pragma unroll
    for (int i = 0; i < 6; ++i) s[i] = so[i] + inc[i];
    if (PLASTIC) {
        // J2 radial return, linear isotropic hardening (no reference
        // counterpart; the elastic instantiation omits it).
        const double pm = div_by((s[0] + s[1]) + s[2], 3.0, 1.0 / 3.0);
        const double d0 = s[0] - pm, d1 = s[1] - pm, d2 = s[2] - pm;
        const double j2 = 0.5 * ((d0 * d0 + d1 * d1) + d2 * d2) + ((s[3] * s[3] + s[4] * s[4]) + s[5] * s[5]);
        const double seq = sqrt(3.0 * j2);
        const double ep_old = S.eps[si];
        const double sy = M.yield0 + M.hardening * ep_old;
        if (seq > sy) {
            const double dl = (seq - sy) / (3.0 * G + M.hardening);
            const double r = 1.0 - 3.0 * G * dl / seq;
            s[0] = d0 * r + pm;
            s[1] = d1 * r + pm;
            s[2] = d2 * r + pm;
            s[3] = s[3] * r;
            s[4] = s[4] * r;
            s[5] = s[5] * r;
            if (!INIT) O.eps[oi] = ep_old + dl;
        }
    }
    if (!INIT) {
#pragma unroll
        for (int i = 0; i < 6; ++i) O.sig[i * os + oi] = s[i];
    }
    const double V0 = S.vol0[si];
    const double Vc = J * V0;
    {
        double w = 0.0;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double sm = 0.5 * (so[i] + s[i]);
            w = w + (i < 3 ? 1.0 : 2.0) * sm * eps[i];
        }
        e_int += w * Vc;
    }
    // hourglass coefficients and history (:1038-1050); Gq = QIA + CR HIA
    const double r43 = 4.0 / 3.0;
    const double r1s8 = 1.0 / sqrt(8.0);
    const double DR = M.c_dr * (r43 * G + M.K) * 0.1 * nx2 * Vc * r1s8 * dt1;
    const double CR = M.c_cr * M.rho * V0 / Vc * S.cb2[si] * M.wos / 4.0;
    double Gq[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const double q = __fma_rn(DR, HIA[i][kk], S.qia[(4 * i + kk) * ss + si]);
            if (!INIT) O.qia[(4 * i + kk) * os + oi] = q;
            Gq[i][kk] = __fma_rn(CR, HIA[i][kk], q);
        }
    // bulk viscosity pressure (:1073-1109)
    const bool visc = !(fabs(vr) < 1.0e-10);
    double pv = 0.0;
    if (visc) {
        const double rho_c = M.rho / J;
        const double l0 = S.cb[si];
        const double m0 = vr < 0.0 ? vr : 0.0;
        pv = rho_c * l0 * (M.cvisq * M.cvisq * l0 * vr * m0 - M.cvisl * M.wos * vr);
        e_vis += -(pv * Vc * vr) * dt1;
    }
    // Z = Vc F^-1 (sigma - p I) - W^T, W = Gq TX
    const double Sp[3][3] = {{s[0] - pv, s[3], s[4]}, {s[3], s[1] - pv, s[5]}, {s[4], s[5], s[2] - pv}};
    double W[3][3], Z[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            W[i][c] = __fma_rn(Gq[i][3], TX[3][c],
                               __fma_rn(Gq[i][2], TX[2][c], __fma_rn(Gq[i][1], TX[1][c], Gq[i][0] * TX[0][c])));
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            Z[c][i] = Vc * __fma_rn(Fi[c][2], Sp[2][i], __fma_rn(Fi[c][1], Sp[1][i], Fi[c][0] * Sp[0][i])) - W[i][c];
    // hourglass power sum_j h_j . v_j = Gq : HIA
    {
        double hp = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) hp = __fma_rn(Gq[i][kk], HIA[i][kk], hp);
        e_hg += hp * dt1;
    }
    // nodal forces f_j = -(B0_j Z) - Gamma_j Gq^T
    // (= -b_j sigma V - h_j + p b_j V: :985-997, :1070, :1106).  Gamma_j Gq^T is
    // summed over the four hourglass vectors in order, nodes with the same
    // leading signs (or the opposite ones) sharing their partial sums; B0_j Z
    // is evaluated once for two opposite corners.
    {
        B0Rows<BT9, SMEM> Bf;
        // (the force array is looked up here: a batch reads it from the stage)
        double* fe = static_cast<double*>(E.fe);
        const int64_t row = E.slot_major ? N.nn_pad : E.ne_pad;
        const bool mapped = REC && E.rows != nullptr;
        const uint32_t rows = mapped ? __ldg(E.rows + e) : 0u;
        auto store = [&](int j, const double (&f)[3]) {
            const int64_t i = E.slot_major ? static_cast<int64_t>(ldin<SMEM>(S.conn + j * ss + si)) : e;
            const int k = mapped ? static_cast<int>((rows >> (4 * j)) & 7u) : j;
            *reinterpret_cast<double2*>(force_xy(fe, row, k, i)) = make_double2(f[0], f[1]);
            *force_z(fe, row, k, i) = f[2];
        };
        if constexpr (BT9) {
            Bf.load(S);
            double f[8][3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double g0 = Gq[i][0], g1 = Gq[i][1], g2 = Gq[i][2], g3 = Gq[i][3];
                const double d = g0 - g1, q = g0 + g1;
                const double dm = d - g2, dp = d + g2, qm = g2 - q, qp = q + g2;
                const double t[8] = {dm - g3, qm + g3, qp - g3, g3 - dp, qp + g3, -(dp + g3), dm + g3, qm - g3};
                double bz[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    bz[j] = __fma_rn(Bf.r[j][2], Z[2][i], __fma_rn(Bf.r[j][1], Z[1][i], Bf.r[j][0] * Z[0][i]));
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j][i] = (Bf.minus(j) ? bz[Bf.index(j)] : -bz[Bf.index(j)]) - t[j];
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) store(j, f[j]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                double bb[3], f[3];
                Bf.row(S, j, bb);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    double tg = gamma_plus(0, j) ? Gq[i][0] : -Gq[i][0];
#pragma unroll
                    for (int kk = 1; kk < 4; ++kk) tg = gamma_plus(kk, j) ? tg + Gq[i][kk] : tg - Gq[i][kk];
                    f[i] = -__fma_rn(bb[2], Z[2][i], __fma_rn(bb[1], Z[1][i], bb[0] * Z[0][i])) - tg;
                }
                store(j, f);
            }
        }
    }
    // compute_dtStable (:828-834)
    {
        const double cd = M.wos, rcd = M.mc.inv_wos;
        const double m0 = vr < 0.0 ? vr : 0.0;
        const double xi = M.cvisl - div_by(M.cvisq * M.cvisq * len, cd, rcd) * m0;
        dts = div_by((sqrt(1.0 + xi * xi) - xi) * len, cd, rcd);
    }
    if (!isfinite(dts)) bad |= ST_NONFINITE;
}

// Element pass: add_inForce_to_rhs's element loop body
// (exDyna3D.cpp:556-573): kinematics, Jaumann stress (+ J2 return),
// hourglass, bulk viscosity, element dt and min edge.  Writes the element's
// 8x3 nodal forces to fe for the node-centric gather.  Every value is the same
// expression, in the same order, as the CPU restatement (explicit fma only).
//
// One element per thread from global memory: the init force pass, and every pass
// over caller-owned rows (ensc_step_noalloc).  Cycles over tiles run
// k_element_fp64_warp.
template <bool PLASTIC, bool INIT, bool BT9, bool TILED>
__global__ void __launch_bounds__(kElemThreads, ENSC_ELEM_MINB_FP64) k_element(ElemArrays E, NodeArrays N, Material M, Ctl* ctl,
                                                             Partials P) {
    if (ctl->done) return;
    const double dt1 = INIT ? 0.0 : ctl->dt_i_1;
    const int64_t ne = E.ne;
    double e_int = 0.0, e_hg = 0.0, e_vis = 0.0;
    double dts_min = DBL_MAX, len_min = DBL_MAX;
    int32_t bad = 0;

    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const int64_t e_end = (ne + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t e0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e0 < e_end; e0 += stride) {
        const bool live = e0 < ne;
        const int64_t e = live ? e0 : 0;
        double dts = DBL_MAX, len = DBL_MAX;
        if (live)
            element_body<PLASTIC, INIT, BT9, TILED>(E, N, M, fp64_src_global<TILED>(E, e), fp64_out_global<TILED>(E, e), dt1, e,
                                             dts, len, e_int, e_hg, e_vis, bad);
        dts_min = dts < dts_min ? dts : dts_min;
        len_min = len < len_min ? len : len_min;
    }
    if (bad) atomicOr(&ctl->status, bad);
    block_min2<kElemThreads>(dts_min, len_min, &ctl->dts_next, &ctl->len_min);
    if (!INIT) {
        double v3[3] = {e_int, e_hg, e_vis};
        block_sum<kElemThreads, 3, 7u>(v3, P.elem, P.n_elem_blocks, blockIdx.x);
    }
}

// The force of one node from per-element forces (E.slot_major 0): the
// caller-owned table of one element per slot, or the general lists, sorted by
// (slot, element): each slot's contributions are summed first (the reference's
// per-slot += in element order), then added to the running total.
__device__ __forceinline__ void listed_forces(const ElemArrays& E, const NodeArrays& N, const int64_t n,
                                              double (&f)[3]) {
    const int64_t np = N.nn_pad, ep = E.ne_pad;
    const double* fe = static_cast<const double*>(E.fe);
    auto at = [&](int k, uint32_t el, double (&r)[3]) {
        const double2 xy = *reinterpret_cast<const double2*>(force_xy(fe, ep, k, el));
        r[0] = xy.x;
        r[1] = xy.y;
        r[2] = *force_z(fe, ep, k, el);
    };
    f[0] = f[1] = f[2] = 0.0;
    if (N.csr_ptr == nullptr) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t el = __ldg(N.ell + k * np + n);
            if (el != ENSC_NONE) {
                double r[3];
                at(k, el, r);
#pragma unroll
                for (int c = 0; c < 3; ++c) f[c] = f[c] + r[c];
            }
        }
        return;
    }
    const int64_t b = N.csr_ptr[n], t = N.csr_ptr[n + 1];
    int cur = -1;
    double sl[3] = {0.0, 0.0, 0.0};
    for (int64_t i = b; i < t; ++i) {
        const uint32_t ent = N.csr_ent[i];
        const int k = static_cast<int>(ent & 7u);
        double r[3];
        at(k, ent >> 3, r);
        if (k != cur) {
            if (cur >= 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) f[c] = f[c] + sl[c];
            }
            cur = k;
#pragma unroll
            for (int c = 0; c < 3; ++c) sl[c] = 0.0 + r[c];
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) sl[c] = sl[c] + r[c];
        }
    }
    if (cur >= 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = f[c] + sl[c];
    }
}

// One node of the node pass where the forces are per element; shared by the
// single-instance, batched and resident-run kernels (KIN: sum the kinetic
// energy).
template <bool KIN = true>
__device__ __forceinline__ void node_body(const ElemArrays& E, const NodeArrays& N, const Material& M,
                                          const double dt_i, const double dt_i_1, const double amp, const int64_t n, double& kin,
                                          double& wext, int32_t& bad) {
    const int64_t np = N.nn_pad;
    const double half = (dt_i + dt_i_1);
    const double dt_avg = (dt_i + dt_i_1) / 2.0;

    double f[3];
    listed_forces(E, N, n, f);
    const double im = N.inv_mass[n];
    const uint32_t code = N.bc[n];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double a = f[c];
        double g = 0.0;
        if (M.gravity_on) {
            g = amp * M.gravity_value * M.gravity_dir[c] / im;  // apply_gravity (:809-824)
            a = a + g;
        }
        const uint32_t cc = (code >> (2 * c)) & 3u;
        double r = 0.0, rf = 0.0;
        if (cc & 2u) {
            r = -a;
            a = 0.0;
        }
        if ((cc & 1u) && a != 0.0) {
            rf = -a;
            r = -a;
            a = 0.0;
        }
        if (cc) N.rf[c * np + n] = rf;
        a = a * im;
        double *pv = node_v64(N, c, n), *pu = node_u64(N, c, n), *px = node_x(N, c, n);
        const double vo = *pv;
        const double vn = vo + half * a / 2.0;
        *pv = vn;
        *pu = *pu + dt_i * vn;
        *px = *px + dt_i * vn;
        const double vb = 0.5 * (vo + vn);
        wext = wext + (g + r) * dt_avg * vb;
        if (KIN) kin = kin + 0.5 * (vn * vn) / im;
        if (!isfinite(vn)) bad |= ST_NONFINITE;
    }
}

// ---- warp-pipelined element pass ---------------------------------------
// Every warp runs its own pipeline over tiles of 32 consecutive elements: two
// shared-memory stages, each filled by one bulk copy of a whole tile while
// the other is computed, and no block-wide barrier per tile.  element_body's
// arithmetic, so results are bit-identical to the other FP64 element passes.
constexpr int kF64PipeWarps = ENSC_F64_PIPE_WARPS;
template <typename L>
constexpr size_t f64_pipe_smem() {
    return static_cast<size_t>(kF64PipeWarps) * (2 * L::kBytes + 16);
}

// Lane 0: the tile at src into shared memory at dst, completing on bar
// (elastic instances leave out eps_p, the tile's last row).
template <bool PLASTIC, typename L>
__device__ __forceinline__ void f64_tile_issue(const void* src, uint32_t dst, uint32_t bar) {
    constexpr uint32_t bytes = PLASTIC ? L::kBytes : L::kEps;
    mbar_arrive_expect_tx(bar, bytes);
    fence_proxy_async_smem();  // the warp's reads of this stage come before the copy into it
    bulk_g2s(dst, src, bytes, bar);
}

template <bool PLASTIC, bool BT9>
__global__ void __launch_bounds__(32 * kF64PipeWarps, ENSC_F64_PIPE_MINB)
    k_element_fp64_warp(ElemArrays E, NodeArrays N, Material M, Ctl* ctl, Partials P) {
    using L = std::conditional_t<BT9, Fp64Tile9, Fp64Tile24>;
    cycle_kernel_enter();
    if (ctl->done) return;
    extern __shared__ __align__(128) unsigned char smem[];
    const double dt1 = ctl->dt_i_1;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    unsigned char* wst = smem + static_cast<size_t>(wid) * 2 * L::kBytes;
    const uint32_t stage0 = smem_addr(wst);
    const uint32_t bar0 = smem_addr(smem + static_cast<size_t>(kF64PipeWarps) * 2 * L::kBytes) + 16u * wid;
    const unsigned char* tiles = reinterpret_cast<const unsigned char*>(E.conn);
    const int ntiles = static_cast<int>((E.ne + 31) / 32);
    const int wstride = static_cast<int>(gridDim.x) * kF64PipeWarps;
    const int w0 = static_cast<int>(blockIdx.x) * kF64PipeWarps + wid;
    if (lane == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
        for (int s = 0; s < 2; ++s) {
            const int t = w0 + s * wstride;
            if (t < ntiles) f64_tile_issue<PLASTIC, L>(tiles + static_cast<int64_t>(t) * L::kBytes, stage0 + s * L::kBytes, bar0 + 8 * s);
        }
    }
    __syncwarp();
    double e_int = 0.0, e_hg = 0.0, e_vis = 0.0;
    double dts_min = DBL_MAX, len_min = DBL_MAX;
    int32_t bad = 0;
    bool timed_out = false;
    int it = 0;
    for (int t = w0; t < ntiles; t += wstride, ++it) {
        const int s = it & 1;
        const uint32_t bar = bar0 + 8 * s;
        const bool ok = mbar_wait_bounded(bar, (it >> 1) & 1);
        if (__any_sync(0xffffffffu, !ok)) {
            timed_out = true;
            break;
        }
        const int e = t * 32 + lane;
        if (e < E.ne) {
            unsigned char* g = const_cast<unsigned char*>(tiles) + static_cast<int64_t>(t) * L::kBytes;
            double dts, len;
            element_body<PLASTIC, false, BT9, true, true, ENSC_F64_PREFETCH>(E, N, M, fp64_src_tile<L>(wst + s * L::kBytes, lane),
                                                                       fp64_out_tile<L>(g, lane), dt1, e, dts, len,
                                                                       e_int, e_hg, e_vis, bad);
            dts_min = dts < dts_min ? dts : dts_min;
            len_min = len < len_min ? len : len_min;
        }
        __syncwarp();  // all lanes are done with stage s
        const int tn = t + 2 * wstride;
        if (lane == 0 && tn < ntiles) f64_tile_issue<PLASTIC, L>(tiles + static_cast<int64_t>(tn) * L::kBytes, stage0 + s * L::kBytes, bar);
    }
    if (timed_out) {
        // record the failure and let the copies this warp started land
        // (bounded) before the block's shared memory is released
        if (lane == 0) {
            atomicOr(&ctl->status, ST_TIMEOUT);
            for (int k = 0; k < 2; ++k) {
                const int itk = it + k;
                if (w0 + itk * wstride < ntiles) mbar_wait_bounded(bar0 + 8 * (itk & 1), (itk >> 1) & 1);
            }
        }
        __syncwarp();
    }
    if (bad) atomicOr(&ctl->status, bad);
    block_min2<32 * kF64PipeWarps>(dts_min, len_min, &ctl->dts_next, &ctl->len_min);
    double v3[3] = {e_int, e_hg, e_vis};
    block_sum<32 * kF64PipeWarps, 3, 7u>(v3, P.elem, P.n_elem_blocks, blockIdx.x);
}

// W consecutive nodes of the node pass where the force rows are by node.  Every
// row is added, empty ones as the zeros they hold, as the reference adds all 8
// slot vectors: the rows start zeroed and only the row's element writes them.
// Nodes at or past nn (row padding) are loaded and stored back unchanged.
//
// pre (resident runs): the nodes' own records, loaded while the grid still works
// on the forces; such a run sums its kinetic energy once, at its end.
template <int W>
struct NodeRowsF64 {
    double im[W], rim[W], q0[W][4], q1[W][4], vz[W];  // rim: 1 / im, under gravity
    uint32_t code;
};
template <int W>
__device__ __forceinline__ void node_rows_load(const NodeView& N, const int64_t n0, NodeRowsF64<W>& r) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
        ld_rec(N.x + 4 * (n0 + j), r.q0[j]);
        ld_rec(N.u + 4 * (n0 + j), r.q1[j]);
    }
    ld_row<W>(static_cast<const double*>(N.v) + n0, r.vz);
    ld_row<W>(N.inv_mass + n0, r.im);
    r.code = ld_bytes<W>(N.bc + n0);
}

// The forces of W consecutive nodes, added up in row order.  MERGE: where a node
// repeats a slot (bit k of its merge byte: row k holds the slot of row k - 1),
// that slot's rows are summed first, as the reference adds each element to its
// slot's vector before it adds the vectors.
template <int W, bool MERGE = false>
__device__ __forceinline__ void node_forces(const NodeView& N, const int64_t n0, double (&f)[3][W]) {
    const int64_t np = N.np;
    const double* fe = static_cast<const double*>(N.fe);
    const uint32_t merge = MERGE ? ld_bytes<W>(N.merge + n0) : 0u;
    double sl[3][W];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int j = 0; j < W; ++j) f[c][j] = sl[c][j] = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        double xy[2 * W], z[W];
        ld_row<2 * W>(force_xy(fe, np, k, n0), xy);
        ld_row<W>(force_z(fe, np, k, n0), z);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const double r[3] = {xy[2 * j], xy[2 * j + 1], z[j]};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if constexpr (MERGE) {
                    const bool same = (merge >> (8 * j + k)) & 1u;
                    f[c][j] = same ? f[c][j] : f[c][j] + sl[c][j];
                    sl[c][j] = (same ? sl[c][j] : 0.0) + r[c];
                } else {
                    f[c][j] = f[c][j] + r[c];
                }
            }
        }
    }
    if constexpr (MERGE)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int j = 0; j < W; ++j) f[c][j] = f[c][j] + sl[c][j];
}

// PRE: rows and forces come in pre and fpre.
template <int W, bool PRE = false, bool MERGE = false>
__device__ __forceinline__ void node_group(const NodeView& N, const double dt_i, const double dt_i_1, const double amp,
                                           const int64_t n0, double& kin, double& wext, int32_t& bad,
                                           const NodeRowsF64<W>* pre = nullptr,
                                           const double (*fpre)[W] = nullptr) {
    const int64_t np = N.np, nn = N.nn;
    const double half = (dt_i + dt_i_1);
    const double dt_avg = (dt_i + dt_i_1) / 2.0;
    NodeRowsF64<W> own;
    if constexpr (PRE) own = *pre;
    else node_rows_load<W>(N, n0, own);
    double f[3][W];
    if constexpr (PRE) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int j = 0; j < W; ++j) f[c][j] = fpre[c][j];
    } else {
        node_forces<W, MERGE>(N, n0, f);
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (n0 + j >= nn) continue;
        const double im = own.im[j];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double* pv = c == 2 ? &own.vz[j] : &own.q1[j][2 + c];
            double* pu = c == 0 ? &own.q0[j][3] : &own.q1[j][c - 1];
            double a = f[c][j];
            double g = 0.0;
            if (N.gravity_on) {
                const double w = amp * N.gravity_value * N.gravity_dir[c];
                if constexpr (PRE) g = div_by(w, im, own.rim[j]);
                else g = w / im;
                a = a + g;
            }
            const uint32_t cc = (own.code >> (8 * j + 2 * c)) & 3u;
            double r = 0.0, rf = 0.0;
            if (cc & 2u) {
                r = -a;
                a = 0.0;
            }
            if ((cc & 1u) && a != 0.0) {
                rf = -a;
                r = -a;
                a = 0.0;
            }
            if (cc) N.rf[c * np + n0 + j] = rf;
            a = a * im;
            const double vo = *pv, vn = vo + half * a / 2.0;
            *pv = vn;
            *pu = *pu + dt_i * vn;
            own.q0[j][c] = own.q0[j][c] + dt_i * vn;
            const double vb = 0.5 * (vo + vn);
            wext = wext + (g + r) * dt_avg * vb;
            if (!PRE) kin = kin + 0.5 * (vn * vn) / im;
            if (!isfinite(vn)) bad |= ST_NONFINITE;
        }
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
        st_rec(N.x + 4 * (n0 + j), own.q0[j]);
        st_rec(N.u + 4 * (n0 + j), own.q1[j]);
    }
    st_row<W>(static_cast<double*>(N.v) + n0, own.vz);
}

// ---- output: the last cycle's acceleration --------------------------------
// solution_a as compute_a leaves it (exDyna3D.cpp:642-644) in the last cycle
// -- assembled element forces, gravity, the acceleration boundary conditions,
// times the inverse mass -- which output_results writes (:231).  The node
// pass does not store it; this pass evaluates it again from the element
// forces that the last force pass left in fe, with the node pass's
// arithmetic in the node pass's order (the grouped layout adds all 8 slots,
// empty ones as the zeros they hold).  Writes interleaved xyz per node.
__global__ void __launch_bounds__(kNodeThreads) k_acceleration(ElemArrays E, NodeArrays N, Material M, const Ctl* ctl,
                                                               double* a_out) {
    const double amp = (M.gravity_on && M.amp_n > 0) ? gravity_amplitude(M.amp, M.amp_n, ctl->time, ctl->dt_i) : 1.0;
    const NodeView nv = node_view(E, N, M, nullptr);
    for (int64_t n = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; n < N.nn;
         n += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        double f[3];
        if (E.slot_major) {
            double g[3][1];
            if (N.merge) node_forces<1, true>(nv, n, g);
            else node_forces<1>(nv, n, g);
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] = g[c][0];
        } else {
            listed_forces(E, N, n, f);
        }
        const double im = N.inv_mass[n];
        const uint32_t code = N.bc[n];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double a = f[c];
            if (M.gravity_on) a = a + amp * M.gravity_value * M.gravity_dir[c] / im;
            const uint32_t cc = (code >> (2 * c)) & 3u;
            if (cc & 2u) a = 0.0;
            if ((cc & 1u) && a != 0.0) a = 0.0;
            a_out[3 * n + c] = a * im;
        }
    }
}

// Node pass: gather of the element forces in slot order (the reference's
// ((((((a0+a1)+a2)+a3)+a4)+a5)+a6)+a7, exDyna3D.cpp:638-639), gravity
// (:819-824), boundary conditions on a (:2029-2145), a = f M^-1 (:642-644),
// v += (dt_i + dt_i_1) a / 2, u += dt_i v, x += dt_i v (:646-654, :688-696).
// MERGE: nodes repeat slots (ElemArrays::rows).
template <bool MERGE>
__global__ void __launch_bounds__(kNodeThreads, ENSC_NODE_MINB_FP64) k_node(ElemArrays E, NodeArrays N, Material M, Ctl* ctl, Partials P) {
    cycle_kernel_enter();
    if (ctl->done) return;
    // stable dt of this cycle (update_minVertex_perMaterial_and_dt :673-679)
    double dt_i;
    const double dt_i_1 = ctl->dt_i_1;
    if (ctl->dt_final) {
        dt_i = ctl->dt_i;
    } else {
        const double lmin = bits_ord(ctl->len_min);
        double d = lmin / ctl->wos;
        const double tmp = ctl->dts_cur;
        d = d < tmp ? d : tmp;
        dt_i = d * ctl->factor;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!(dt_i > 0.0) || !isfinite(dt_i)) atomicOr(&ctl->status, ST_BAD_DT);
        if (!ctl->dt_final) ctl->dt_i = dt_i;
        ctl->cycles_done += 1;
        ctl->energy_pending = 1;
    }
    const int64_t nn = N.nn;
    const double amp = (M.gravity_on && M.amp_n > 0) ? gravity_amplitude(M.amp, M.amp_n, ctl->time, dt_i) : 1.0;
    double kin = 0.0, wext = 0.0;
    int32_t bad = 0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (E.slot_major && E.tile_bytes) {
        constexpr int W = kNodeGroupFp64;
        const NodeView nv = node_view(E, N, M, ctl);
        // from the last nodes back: their forces are the latest in L2, and the
        // first nodes' records stay there for the next element pass (B200,
        // 2,097,152 elements: 3% of a mixed cycle, 2% of an FP64 one)
        const int64_t ng = (nn + W - 1) / W;
        for (int64_t g = t0; g < ng; g += stride)
            node_group<W, false, MERGE>(nv, dt_i, dt_i_1, amp, (ng - 1 - g) * W, kin, wext, bad);
    } else {
        for (int64_t n = t0; n < nn; n += stride) node_body(E, N, M, dt_i, dt_i_1, amp, n, kin, wext, bad);
    }
    if (bad) atomicOr(&ctl->status, bad);
    double v2[2] = {kin, wext};
    block_sum<kNodeThreads, 2, 2u>(v2, P.node, P.n_node_blocks, blockIdx.x);
}

// ---- resident runs (ensc_run.cuh) -----------------------------------------
// 8 warps per SM as in the warp-pipelined pass; a tile takes 8,960 bytes, so
// that 25 tiles fit an SM and 148 SMs hold 113,664 elements at three tiles per
// warp.  (Only for B0 in its 9-number form, which every mesh whose constants
// are computed here has.)
constexpr int kRunWarpsF64 = 8;
template <bool PLASTIC>
struct RunFp64 {
    using L = Fp64Tile9;
    static constexpr uint32_t kTileBytes = L::kBytes;
    static constexpr bool kKinInUpdate = false;  // velocities are stored as they are computed
    __device__ static const uint32_t* conn(const unsigned char* tile) {
        return reinterpret_cast<const uint32_t*>(tile);
    }
    __device__ static void load_tile(const ElemArrays& E, uint32_t dst, uint32_t bar, int64_t t, int lane) {
        if (lane == 0)
            f64_tile_issue<PLASTIC, L>(reinterpret_cast<const unsigned char*>(E.conn) + t * L::kBytes, dst, bar);
    }
    __device__ static void store_tile(const ElemArrays& E, const unsigned char* tile, int64_t t, int lane) {
        // whole rows: the entries past ne are padding
        unsigned char* g = const_cast<unsigned char*>(reinterpret_cast<const unsigned char*>(E.conn)) + t * L::kBytes;
        constexpr uint32_t end = PLASTIC ? L::kBytes : L::kEps;
        for (uint32_t o = L::kState + 8u * lane; o < end; o += 256)
            *reinterpret_cast<double*>(g + o) = *reinterpret_cast<const double*>(tile + o);
    }
    __device__ static void element(const ElemArrays& E, const NodeArrays& N, const Material& M, unsigned char* tile,
                                   double dt1, int64_t e, int lane, double& dts, double& len, double& e_int,
                                   double& e_hg, double& e_vis, int32_t& bad) {
        element_body<PLASTIC, false, true, true, true, ENSC_F64_PREFETCH>(E, N, M, fp64_src_tile<L>(tile, lane),
                                                                    fp64_out_tile<L>(tile, lane), dt1, e, dts, len,
                                                                    e_int, e_hg, e_vis, bad);
    }
    // W nodes per thread, their rows loaded ahead of the forces; a thread's
    // further nodes (meshes with more than 2 per thread) load both together.
    // Meshes with node lists read them node by node.
    template <int W>
    struct Nodes {
        NodeRowsF64<W> rows;
        double f[3][W];
        __device__ void load(const ElemArrays& E, const NodeArrays& N, const Material& M, int64_t t0) {
            if (E.slot_major && t0 * W < N.nn) {
                node_rows_load<W>(node_view(E, N, M, nullptr), t0 * W, rows);
                if (M.gravity_on) reciprocals();
            }
        }
        __device__ void reciprocals() {
#pragma unroll
            for (int j = 0; j < W; ++j) rows.rim[j] = 1.0 / rows.im[j];
        }
        __device__ void forces(const NodeView& nv, int64_t n0) {
            if (nv.merge) node_forces<W, true>(nv, n0, f);
            else node_forces<W>(nv, n0, f);
        }
        __device__ void gather(const ElemArrays& E, const NodeArrays& N, const Material& M, int64_t t0) {
            if (E.slot_major && t0 * W < N.nn) forces(node_view(E, N, M, nullptr), t0 * W);
        }
        __device__ void update(const ElemArrays& E, const NodeArrays& N, const Material& M, double dt_i, double dt_i_1,
                               double amp, int64_t t0, int64_t stride, double& wext, int32_t& bad) {
            double kin = 0.0;
            if (E.slot_major) {
                const NodeView nv = node_view(E, N, M, nullptr);
                if (t0 * W < N.nn) node_group<W, true>(nv, dt_i, dt_i_1, amp, t0 * W, kin, wext, bad, &rows, f);
                if (W > 1)
                    for (int64_t g = t0 + stride; g * W < N.nn; g += stride) {
                        node_rows_load<W>(nv, g * W, rows);
                        if (M.gravity_on) reciprocals();
                        forces(nv, g * W);
                        node_group<W, true>(nv, dt_i, dt_i_1, amp, g * W, kin, wext, bad, &rows, f);
                    }
            } else {
                for (int64_t n = t0; n < N.nn; n += stride)
                    node_body<false>(E, N, M, dt_i, dt_i_1, amp, n, kin, wext, bad);
            }
        }
    };
    __device__ static double kinetic(const NodeArrays& N, int64_t n) {
        double kin = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double v = *node_v64(N, c, n);
            kin = kin + 0.5 * (v * v) / N.inv_mass[n];
        }
        return kin;
    }
};

template <bool PLASTIC, bool CLUSTER, int W>
__global__ void __launch_bounds__(32 * kRunWarpsF64, 1)
    k_run_fp64(ElemArrays E, NodeArrays N, Material M, Ctl* ctl, Partials P, RunSync* sync, RunArgs a) {
    run_cycles<RunFp64<PLASTIC>, CLUSTER, W>(E, N, M, ctl, P, sync, a);
}

// ---- batched instances --------------------------------------------------------
// Element tiles of 32 elements and node tiles of 32 * kNodeGroupFp64 nodes,
// each inside one instance whose arrays, material and control block come from
// the instance table.  The element pass runs one pipeline per warp over the
// tile list; the node
// pass gives each node tile to one warp.  Work terms add up across cycles in a
// partial slot per node tile and per run of element tiles (below), one owner per
// slot and pass; a node tile keeps its latest kinetic energy.  k_fold_batch folds
// them per instance in tile order.  Arithmetic per element and node is that of
// the single-instance kernels, so states are bit-identical to them; the element
// sums are grouped by the grid, so their last bits may change with it.
// A batch stage: a tile, then its instance descriptor, its element-pass scalars
// (StageHdr), the TileInfo the filling lane writes, and the ETileSrc record of
// the tile that uses the stage next (as in the mixed batch pass).  The tile's
// room is T.tile_room: 8,960 bytes, or 12,800 while the batch holds an
// instance with its own 24-number B0^T.

// Lane 0 of a warp fills a stage.
__device__ __forceinline__ void f64_batch_issue(const BatchTables& T, const ETileSrc& src, int64_t t_next,
                                                int64_t ntiles, unsigned char* stage, uint32_t dst, uint32_t bar) {
    const bool next = t_next < ntiles;
    const uint32_t o = static_cast<uint32_t>(T.tile_room);
    TileInfo* ti = reinterpret_cast<TileInfo*>(stage + o + kBatchInfoOff);
    ti->slot = src.slot;
    ti->base = src.base;
    mbar_arrive_expect_tx(bar, static_cast<uint32_t>(src.bytes) + sizeof(InstanceDesc) + sizeof(StageHdr) +
                                   (next ? sizeof(ETileSrc) : 0u));
    fence_proxy_async_smem();  // the warp's reads of this stage come before the copies into it
    bulk_g2s(dst, src.tile, static_cast<uint32_t>(src.bytes), bar);
    bulk_g2s(dst + o, T.desc + src.slot, sizeof(InstanceDesc), bar);
    bulk_g2s(dst + o + kBatchHdrOff, T.sparam + src.slot, sizeof(StageHdr), bar);
    if (next) bulk_g2s(dst + o + kBatchNextOff, T.etile_src + t_next, sizeof(ETileSrc), bar);
}

// The batched FP64 element pass: one pipeline per warp over tiles of 32
// elements, element_body's arithmetic per element, so states are bit-identical
// to the single-instance pass.  Sums are kept over a warp's consecutive tiles of
// one instance and reduced into the partial slot of the first: reducing per tile
// took 3% more of a 24-instance sweep's cycle.
__global__ void __launch_bounds__(32 * kF64PipeWarps, ENSC_F64_PIPE_MINB) k_element_batch_fp64(BatchTables T) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t SB = static_cast<uint32_t>(T.tile_room) + kBatchTailBytes;
    unsigned char* wst = smem + static_cast<size_t>(wid) * 2 * SB;
    const uint32_t stage0 = smem_addr(wst);
    const uint32_t bar0 = smem_addr(smem + static_cast<size_t>(kF64PipeWarps) * 2 * SB) + 16u * wid;
    cycle_kernel_enter();
    const int ntiles = T.counts[0];
    const int wstride = static_cast<int>(gridDim.x) * kF64PipeWarps;
    const int w0 = static_cast<int>(blockIdx.x) * kF64PipeWarps + wid;
    if (lane == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
        for (int s = 0; s < 2; ++s) {
            const int t = w0 + s * wstride;
            if (t < ntiles)
                f64_batch_issue(T, T.etile_src[t], t + 2 * wstride, ntiles, wst + s * SB, stage0 + s * SB, bar0 + 8 * s);
        }
    }
    __syncwarp();
    bool timed_out = false;
    int it = 0;
    int t = w0;
    // the current run, consecutive tiles of one instance: its slot, first tile and sums
    int run_slot = -1, run_tile = 0;
    bool live = false;
    double ei = 0.0, eh = 0.0, ev = 0.0, dts = DBL_MAX, len = DBL_MAX;
    int32_t bad = 0;
    for (; t < ntiles; t += wstride, ++it) {
        const int s = it & 1;
        const uint32_t bar = bar0 + 8 * s;
        const bool ok = mbar_wait_bounded(bar, (it >> 1) & 1);
        if (__any_sync(0xffffffffu, !ok)) {
            timed_out = true;
            break;
        }
        unsigned char* st = wst + s * SB;
        unsigned char* tail = st + T.tile_room;
        const InstanceDesc& d = *reinterpret_cast<const InstanceDesc*>(tail);
        const StageHdr& h = *reinterpret_cast<const StageHdr*>(tail + kBatchHdrOff);
        const TileInfo& ti = *reinterpret_cast<const TileInfo*>(tail + kBatchInfoOff);
        const int slot = ti.slot, e = ti.base + lane;
        if (slot != run_slot) {
            if (live) batch_tile_sums(T, run_tile, run_slot, lane, ei, eh, ev, dts, len, bad);
            ei = eh = ev = 0.0;
            dts = len = DBL_MAX;
            bad = 0;
            run_slot = slot;
            run_tile = t;
            live = h.live != 0;
        }
        if (live && e < d.E.ne) {
            // arrays copied to registers, material read at use
            const ElemArrays E = d.E;
            const NodeArrays N = d.N;
            const double dt1 = h.dt1;
            unsigned char* g = tile_row(E, const_cast<unsigned char*>(reinterpret_cast<const unsigned char*>(E.conn)), ti.base);
            double d1, l1;
            if (E.bt9)
                element_body<true, false, true, true, true, ENSC_F64_PREFETCH>(E, N, d.M, fp64_src_tile<Fp64Tile9>(st, lane),
                                                                         fp64_out_tile<Fp64Tile9>(g, lane), dt1, e, d1, l1, ei, eh,
                                                                         ev, bad);
            else
                element_body<true, false, false, true, true, ENSC_F64_PREFETCH>(E, N, d.M, fp64_src_tile<Fp64Tile24>(st, lane),
                                                                          fp64_out_tile<Fp64Tile24>(g, lane), dt1, e, d1, l1, ei, eh,
                                                                          ev, bad);
            dts = d1 < dts ? d1 : dts;
            len = l1 < len ? l1 : len;
        }
        __syncwarp();  // all lanes are done with stage s
        const int tn = t + 2 * wstride;
        if (lane == 0 && tn < ntiles) {
            const ETileSrc src = *reinterpret_cast<const ETileSrc*>(tail + kBatchNextOff);
            f64_batch_issue(T, src, tn + 2 * wstride, ntiles, st, stage0 + s * SB, bar);
        }
    }
    if (!timed_out) {
        if (live) batch_tile_sums(T, run_tile, run_slot, lane, ei, eh, ev, dts, len, bad);
    } else if (lane == 0) {
        // record the failure on the instance whose tile could not be read and
        // let the copies this warp started land (bounded) before exiting
        atomicOr(&T.ctl[T.etile_inst[t]].status, ST_TIMEOUT);
        for (int k = 0; k < 2; ++k) {
            const int itk = it + k;
            if (w0 + itk * wstride < ntiles) mbar_wait_bounded(bar0 + 8 * (itk & 1), (itk >> 1) & 1);
        }
    }
    element_pass_done(T);
}

// As k_node_batch_mixed: one warp per node tile, slots and first nodes read
// two tiles ahead, table lines prefetched into L1 one tile ahead.
template <int NT>
__global__ void __launch_bounds__(NT, ENSC_NODE_MINB_FP64 * kNodeThreads / NT) k_node_batch_fp64(BatchTables T) {
    constexpr int W = kNodeGroupFp64;
    const int lane = threadIdx.x & 31;
    const int warp = static_cast<int>((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
    const int nwarps = static_cast<int>((static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5);
    cycle_kernel_enter();
    const int ntiles = T.counts[1];
    // from the last tile back, as the single-instance pass (a 48-instance mixed
    // sweep 127.5 to 119.5 us a cycle, 24 FP64 instances 112.5 to 107)
    const int32_t *inst = T.ntile_inst + (ntiles - 1), *first = T.ntile_base + (ntiles - 1);
    int slot = warp < ntiles ? __ldg(inst - warp) : 0;
    int slot_n = warp + nwarps < ntiles ? __ldg(inst - (warp + nwarps)) : 0;
    int base = warp < ntiles ? __ldg(first - warp) : 0;
    int base_n = warp + nwarps < ntiles ? __ldg(first - (warp + nwarps)) : 0;
    for (int t = warp; t < ntiles; t += nwarps) {
        const int t2 = t + 2 * nwarps;
        const int slot_nn = t2 < ntiles ? __ldg(inst - t2) : 0;
        const int base_nn = t2 < ntiles ? __ldg(first - t2) : 0;
        if (lane == 0) {
            prefetch_l1(T.nview + slot_n);
            prefetch_l1(T.nparam + slot_n);
        }
        const NodeParam p = ld_param(T.nparam + slot);
        if (p.live) {
            const NodeView v = ld_view(T.nview + slot);
            const double dt_i = p.dt_i, dt_i_1 = p.dt_i_1, amp = p.amp;
            double kin = 0.0, wext = 0.0;
            int32_t bad = 0;
            const int64_t n0 = static_cast<int64_t>(base) + static_cast<int64_t>(lane) * W;
            if (n0 < v.nn) {
                if (v.grouped && !v.merge) {
                    node_group<W>(v, dt_i, dt_i_1, amp, n0, kin, wext, bad);
                } else if (v.grouped) {
                    node_group<W, false, true>(v, dt_i, dt_i_1, amp, n0, kin, wext, bad);
                } else {
                    const InstanceDesc& d = T.desc[slot];
                    for (int j = 0; j < W && n0 + j < v.nn; ++j)
                        node_body(d.E, d.N, d.M, dt_i, dt_i_1, amp, n0 + j, kin, wext, bad);
                }
            }
            kin = batch_warp_sum(kin);
            wext = batch_warp_sum(wext);
            bad = static_cast<int32_t>(__reduce_or_sync(0xffffffffu, static_cast<unsigned>(bad)));
            if (lane == 0) {
                double* part = T.ntile_part + 2 * static_cast<int64_t>(ntiles - 1 - t);
                if (bad) atomicOr(&v.ctl->status, bad);
                part[0] = kin;
                atomicAdd(part + 1, wext);  // one writer per slot and pass
            }
        }
        slot = slot_n;
        slot_n = slot_nn;
        base = base_n;
        base_n = base_nn;
    }
}

}  // namespace

void launch_element_fp64(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                         int grid, bool init, cudaStream_t st) {
    if (!E.tile_bytes) {  // caller-owned rows (ensc_step_noalloc)
        if (M.plastic) {
            if (init) k_element<true, true, false, false><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl, P);
            else k_element<true, false, false, false><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl, P);
        } else {
            if (init) k_element<false, true, false, false><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl, P);
            else k_element<false, false, false, false><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl, P);
        }
        return;
    }
    auto pick = [&](auto bt9) {
        constexpr bool B9 = decltype(bt9)::value;
        constexpr size_t smem = f64_pipe_smem<std::conditional_t<B9, Fp64Tile9, Fp64Tile24>>();
        if (M.plastic) {
            if (init) k_element<true, true, B9, true><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl, P);
            else launch_cycle_kernel(k_element_fp64_warp<true, B9>, grid, 32 * kF64PipeWarps, smem, st, E, N, M, ctl, P);
        } else {
            if (init) k_element<false, true, B9, true><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl, P);
            else launch_cycle_kernel(k_element_fp64_warp<false, B9>, grid, 32 * kF64PipeWarps, smem, st, E, N, M, ctl, P);
        }
    };
    if (E.bt9) pick(std::true_type{});
    else pick(std::false_type{});
}

void launch_node_fp64(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                      int grid, cudaStream_t st) {
    if (N.merge) k_node<true><<<grid, kNodeThreads, 0, st>>>(E, N, M, ctl, P);
    else k_node<false><<<grid, kNodeThreads, 0, st>>>(E, N, M, ctl, P);
}

int occupancy_element_fp64(bool plastic, bool bt9) {
    // more than the default 48 KB of dynamic shared memory: set on the current
    // device, before any launch or capture
    int nb = 0;
    auto query = [&nb](auto kernel, size_t smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, 32 * kF64PipeWarps, smem);
    };
    if (bt9) {
        if (plastic) query(k_element_fp64_warp<true, true>, f64_pipe_smem<Fp64Tile9>());
        else query(k_element_fp64_warp<false, true>, f64_pipe_smem<Fp64Tile9>());
    } else {
        if (plastic) query(k_element_fp64_warp<true, false>, f64_pipe_smem<Fp64Tile24>());
        else query(k_element_fp64_warp<false, false>, f64_pipe_smem<Fp64Tile24>());
    }
    return nb;
}

void launch_acceleration_fp64(const ElemArrays& E, const NodeArrays& N, const Material& M, const Ctl* ctl,
                              double* a_aos, cudaStream_t st) {
    const int64_t g = std::min<int64_t>((N.nn + kNodeThreads - 1) / kNodeThreads, 65535);
    k_acceleration<<<static_cast<int>(g), kNodeThreads, 0, st>>>(E, N, M, ctl, a_aos);
}

int node_group_width(bool mixed_precision) { return mixed_precision ? kNodeGroupMixed : kNodeGroupFp64; }

int occupancy_node_fp64() {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_node<false>, kNodeThreads, 0);
    return nb;
}


static size_t f64_batch_smem(int tile_room) {
    return static_cast<size_t>(kF64PipeWarps) * (2 * (static_cast<size_t>(tile_room) + kBatchTailBytes) + 16);
}
void launch_element_batch_fp64(const BatchTables& T, int grid, cudaStream_t st) {
    launch_cycle_kernel(k_element_batch_fp64, grid, 32 * kF64PipeWarps, f64_batch_smem(T.tile_room), st, T);
}
void launch_node_batch_fp64(const BatchTables& T, int grid, int threads, cudaStream_t st) {
    if (threads == kNodeThreads / 2) k_node_batch_fp64<kNodeThreads / 2><<<grid, threads, 0, st>>>(T);
    else k_node_batch_fp64<kNodeThreads><<<grid, kNodeThreads, 0, st>>>(T);
}
int occupancy_element_batch_fp64(int tile_room) {
    int nb = 0;
    // dynamic shared memory above the default 48 KB: set on the current
    // device before any launch or capture
    cudaFuncSetAttribute(k_element_batch_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(f64_batch_smem(Fp64Tile24::kBytes)));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_element_batch_fp64, 32 * kF64PipeWarps,
                                                  f64_batch_smem(tile_room));
    return nb;
}

RunPlan plan_run_fp64(int64_t ne, int64_t nn, bool plastic, bool bt9, int sms) {
    if (!bt9) return RunPlan{};
    return plastic ? plan_run(k_run_fp64<true, true, 1>, k_run_fp64<true, true, 2>, k_run_fp64<true, false, 1>,
                              k_run_fp64<true, false, 2>, ne, nn, sms, kRunWarpsF64, RunFp64<true>::kTileBytes)
                   : plan_run(k_run_fp64<false, true, 1>, k_run_fp64<false, true, 2>, k_run_fp64<false, false, 1>,
                              k_run_fp64<false, false, 2>, ne, nn, sms, kRunWarpsF64, RunFp64<false>::kTileBytes);
}
cudaError_t launch_run_fp64(const RunPlan& p, const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl,
                            const Partials& P, RunSync* sync, const RunArgs& a, cudaStream_t st) {
    using K = void (*)(ElemArrays, NodeArrays, Material, Ctl*, Partials, RunSync*, RunArgs);
    static const K kernels[8] = {k_run_fp64<false, false, 1>, k_run_fp64<false, false, 2>, k_run_fp64<false, true, 1>,
                                 k_run_fp64<false, true, 2>,  k_run_fp64<true, false, 1>,  k_run_fp64<true, false, 2>,
                                 k_run_fp64<true, true, 1>,   k_run_fp64<true, true, 2>};
    return launch_run(kernels[(M.plastic ? 4 : 0) + (p.cluster ? 2 : 0) + p.node_width - 1], p, st, E, N, M, ctl, P,
                      sync, a);
}

int occupancy_node_batch_fp64(int threads) {
    int nb = 0;
    if (threads == kNodeThreads / 2)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_node_batch_fp64<kNodeThreads / 2>, threads, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_node_batch_fp64<kNodeThreads>, kNodeThreads, 0);
    return nb;
}

}  // namespace ensc
