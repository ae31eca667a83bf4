// Mixed-precision stepper kernels: the element pass (kinematics, Jaumann /
// J2 stress, hourglass, bulk viscosity) and the force gather run in FP32;
// nodal position accumulation (x += dt v; the displacement is x minus a
// stored reference position), the clock, the stable-dt reduction and the
// energy sums stay FP64.
//
// Same algorithm and data flow as the FP64 path (ensc_fp64.cu); operation
// order is free here (FMA contraction on), accuracy is checked against the
// FP64 path by relative displacement error and energy drift.
//
// Element arrays (MixedTile): the bt rows hold A = sum_j B0_j s_j^T (the
// one-point B0 rows are A s_j / 8, s_j the node's reference-corner signs) as a
// float pair, 9 hi then 9 lo rows; cbrt_v0, sigma, qia, eps_p and fe are float;
// vol0 is double.
// Node arrays: records of x (double) and two velocity components (float), the
// third as a row, with 16-bit residual rows; the u rows hold the reference
// position x - u (double).
#include "ensc_device.cuh"
#include "ensc_kernels.h"
#include "ensc_run.cuh"
#include "ensc_stage.cuh"

#include <cfloat>

namespace ensc {
namespace {

__device__ __forceinline__ float det3f(const float m[3][3]) {
    return m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1]) - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0]) +
           m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
}

__device__ __forceinline__ float cof3f(const float m[3][3], int i, int j) {
    const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
    return m[i1][j1] * m[i2][j2] - m[i1][j2] * m[i2][j1];
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block sum of NV values into out_slots[i * stride + slot]; values whose bit
// is set in ACC are added to the slot (it accumulates over cycles, one writer
// per slot and pass), the others stored.
template <int NT, int NV, unsigned ACC = 0u>
__device__ __forceinline__ void block_sum_d(double (&v)[NV], double* out_slots, int stride, int slot) {
    __shared__ double red[NV][NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const double s = warp_sum_d(v[i]);
        if (lane == 0) red[i][wid] = s;
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double s = lane < NT / 32 ? red[i][lane] : 0.0;
            s = warp_sum_d(s);
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
__device__ __forceinline__ void block_min2_d(double a, double b, unsigned long long* ga, unsigned long long* gb) {
    __shared__ unsigned long long ra[NT / 32], rb[NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long x = ord_bits(a), y = ord_bits(b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long wx = __shfl_xor_sync(0xffffffffu, x, o);
        const unsigned long long wy = __shfl_xor_sync(0xffffffffu, y, o);
        x = wx < x ? wx : x;
        y = wy < y ? wy : y;
    }
    if (lane == 0) {
        ra[wid] = x;
        rb[wid] = y;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < NT / 32; ++i) {
            x = ra[i] < x ? ra[i] : x;
            y = rb[i] < y ? rb[i] : y;
        }
        atomicMin(ga, x);
        atomicMin(gb, y);
    }
    __syncthreads();
}

// Element pass (add_inForce_to_rhs element loop body, exDyna3D.cpp:556-573)
// in FP32.  Node coordinates enter as FP64 offsets from the element's node
// 0; the geometry that every element of a uniform mesh shares (F, edges,
// B0) is carried in FP64 or as float pairs.  Node data are visited twice
// (kinematics, then forces), one component at a time, through the corner
// transforms below.  The hourglass force uses the reassociated sum
// sum_k ATAU(k,j) (QIA(i,k) + CR HIA(i,k))  (exDyna3D.cpp:1053-1070).

// Where one element's inputs are read from and its evolving rows written: a
// tile of 32 elements, in global or shared memory, with the element at `i`.
struct MixedSrc {
    const uint32_t* conn;   // [8] rows
    const float* a;         // [18] rows: A hi (3c+m), then A lo
    const double* vol0;
    const float* cb;
    const float* sig;       // [6] rows
    const float* qia;       // [12] rows
    const float* eps;
    int i;
};
struct MixedOut {
    float* sig;             // [6] rows
    float* qia;             // [12] rows
    float* eps;
    int i;
};
__device__ __forceinline__ MixedSrc mixed_src_tile(const unsigned char* t, int lane) {
    using L = MixedTile;
    return MixedSrc{reinterpret_cast<const uint32_t*>(t),
                    reinterpret_cast<const float*>(t + L::kBt),
                    reinterpret_cast<const double*>(t + L::kVol0),
                    reinterpret_cast<const float*>(t + L::kCb),
                    reinterpret_cast<const float*>(t + L::kSig),
                    reinterpret_cast<const float*>(t + L::kQia),
                    reinterpret_cast<const float*>(t + L::kEps),
                    lane};
}
__device__ __forceinline__ MixedOut mixed_out_tile(unsigned char* t, int lane) {
    using L = MixedTile;
    return MixedOut{reinterpret_cast<float*>(t + L::kSig), reinterpret_cast<float*>(t + L::kQia),
                    reinterpret_cast<float*>(t + L::kEps), lane};
}
// tile t of an instance in global memory
__device__ __forceinline__ unsigned char* mixed_tile(const ElemArrays& E, int64_t t) {
    return const_cast<unsigned char*>(reinterpret_cast<const unsigned char*>(E.conn)) + t * MixedTile::kBytes;
}

// The one-point B0 row of local node j is A s_j / 8 with A = sum_j B0_j s_j^T
// and s_j the node's reference-corner signs (xi, eta, zeta), Element_HexN8.cpp
// :49-91.

// Sums over the 8 nodes with the signs of the reference corners.  Node j sits
// at corner bits x + 2y + 4z (x set where xi = +1, y for eta, z for zeta);
// for a subset S of {xi, eta, zeta} (bits 0, 1, 2) the coefficient
// c[S] = sum_j (prod_{d in S} sigma_d(j)) a_j, sigma_d(j) = +-1.  The corner
// signs are c[1], c[2], c[4]; the hourglass vectors are
// Gamma = (c[3], -c[6], -c[5], c[7]) (xi eta, -eta zeta, -zeta xi,
// xi eta zeta).  One butterfly of 24 additions gives all of them.
template <typename T>
__device__ __forceinline__ void corner_coeffs(const T (&a)[8], T (&c)[8]) {
    constexpr int kBits[8] = {0, 1, 3, 2, 4, 5, 7, 6};
#pragma unroll
    for (int j = 0; j < 8; ++j) c[kBits[j]] = a[j];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!(i & (1 << d))) {
                const T lo = c[i], hi = c[i | (1 << d)];
                c[i] = hi + lo;
                c[i | (1 << d)] = hi - lo;
            }
}

// The other direction: node values a_j = sum_S c[S] prod_{d in S} sigma_d(j)
// (c is overwritten).
template <typename T>
__device__ __forceinline__ void corner_values(T (&c)[8], T (&a)[8]) {
    constexpr int kBits[8] = {0, 1, 3, 2, 4, 5, 7, 6};
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!(i & (1 << d))) {
                const T c0 = c[i], c1 = c[i | (1 << d)];
                c[i | (1 << d)] = c0 + c1;
                c[i] = c0 - c1;
            }
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = c[kBits[j]];
}

// One element of the mixed element pass (see the kernel comment below);
// shared by the single-instance, staged, batched and resident-run kernels.
// Inputs come from S, the evolving rows go to O and the forces to the
// instance's force array at element e.  Node rows are read with plain loads:
// a resident run rewrites them between its cycles.
// FOUT: the 24 nodal forces go to fout[3 * 8] (component-major) instead of
// the instance's force array, for the patch assembly.
template <bool PLASTIC, bool INIT, bool SMEM = false, bool FOUT = false>
__device__ __forceinline__ void element_body_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M,
                                                   const MixedSrc& S, const MixedOut& O, const float dt1,
                                                   const double dt1d, const int64_t e, double& dts, double& len,
                                                   double& e_int, double& e_hg, double& e_vis, int32_t& bad,
                                                   float* fout = nullptr) {
    constexpr int ss = 32, os = 32;
    const int si = S.i, oi = O.i;
    const double* X = N.x;
    const float* V = static_cast<const float*>(N.v);
    const float G = M.mc.G;
    const float lam_hi = M.mc.lam_hi, lam_lo = M.mc.lam_lo;
    const float g2_hi = M.mc.g2_hi, g2_lo = M.mc.g2_lo;
    const float rho = M.mc.rho, wos = M.mc.wos;
    const float cvisl = M.mc.cvisl, cvisq = M.mc.cvisq;
    const float y0 = M.mc.y0, H = M.mc.H;
    const float DRc = M.mc.DRc, CRc = M.mc.CRc;
    if (!FOUT && E.rows) prefetch_l1(E.rows + e);  // read with the forces
    uint32_t nk[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) nk[k] = ldin<SMEM>(S.conn + k * ss + si);
    // the node records, and vz
    double q[8][4];
    float vz[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) ld_rec(X + 4 * static_cast<int64_t>(nk[k]), q[k]);
#pragma unroll
    for (int k = 0; k < 8; ++k) vz[k] = V[nk[k]];
    // coordinates relative to node 0, as FP64 differences, one component at a
    // time: hourglass projections TAU x = TAU (x - x0) (the Gamma rows sum to
    // zero) rounded to FP32; the minimum edge and F = sum_j (x_j - x_0) B0_j
    // = (sum_j (x_j - x_0) s_j^T) A^T / 8 (= I + u_e B0^T, as
    // sum_j X0_j B0_j = I and sum_j B0_j = 0) kept in FP64, since on a
    // uniform mesh the FP32 rounding of the spacing would be the same for
    // every element and shift the stiffness and the stable dt of all of them
    float TX[4][3];
    float F[3][3];
    float Ah[3][3], Al[3][3];
    {
        constexpr int A0[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3};
        constexpr int A1[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
        double e2[12];
        double Gx[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const double xo = q[0][r];
            double xd[8];
            xd[0] = 0.0;
#pragma unroll
            for (int k = 1; k < 8; ++k) xd[k] = q[k][r] - xo;
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                const double d = xd[A1[i]] - xd[A0[i]];
                e2[i] = r == 0 ? d * d : fma(d, d, e2[i]);
            }
            double c[8];
            corner_coeffs(xd, c);
            Gx[r][0] = c[1];
            Gx[r][1] = c[2];
            Gx[r][2] = c[4];
            TX[0][r] = static_cast<float>(c[3]);
            TX[1][r] = static_cast<float>(-c[6]);
            TX[2][r] = static_cast<float>(-c[5]);
            TX[3][r] = static_cast<float>(c[7]);
        }
        // A = sum_j B0_j s_j^T as a float pair (hi + lo); B0 enters every
        // product through A, so no FP32 rounding of the reference geometry is
        // shared by all elements of a uniform mesh
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                Ah[c][m] = ldin<SMEM>(S.a + (3 * c + m) * ss + si);
                Al[c][m] = ldin<SMEM>(S.a + (9 + 3 * c + m) * ss + si);
            }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double t = 0.0;
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    t = fma(Gx[r][m], static_cast<double>(Ah[c][m]) + static_cast<double>(Al[c][m]), t);
                F[r][c] = static_cast<float>(0.125 * t);
            }
        double m = DBL_MAX;
#pragma unroll
        for (int i = 0; i < 12; ++i) m = fmin(m, e2[i]);
        len = sqrt(m);
    }
    const float J = det3f(F);
    if (!(J > 0.f)) bad |= ST_INVERTED;
    const float invdet = 1.f / J;
    float Fi[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Fi[i][j] = cof3f(F, j, i) * invdet;
    // L0 = v_e B0^T = (sum_j v_j s_j^T) A^T / 8, VT = v_e Gamma^T (both from
    // the corner coefficients of each velocity component),
    // NX2 = sum_j |B0_j|^2 = |A|^2 / 8 (sum_j s_j s_j^T = 8 I)
    float L0[3][3], VT[3][4], nx2 = 0.f;
    {
        float Gv[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            float a[8], c[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] = r == 0 ? rec_vx(q[j][3]) : r == 1 ? rec_vy(q[j][3]) : vz[j];
            corner_coeffs(a, c);
            Gv[r][0] = c[1];
            Gv[r][1] = c[2];
            Gv[r][2] = c[4];
            VT[r][0] = c[3];
            VT[r][1] = -c[6];
            VT[r][2] = -c[5];
            VT[r][3] = c[7];
        }
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float t = Gv[r][0] * Al[c][0];
                t = fmaf(Gv[r][1], Al[c][1], t);
                t = fmaf(Gv[r][2], Al[c][2], t);
                t = fmaf(Gv[r][0], Ah[c][0], t);
                t = fmaf(Gv[r][1], Ah[c][1], t);
                t = fmaf(Gv[r][2], Ah[c][2], t);
                L0[r][c] = 0.125f * t;
            }
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int m = 0; m < 3; ++m) nx2 = fmaf(Ah[c][m], Ah[c][m], nx2);
        nx2 *= 0.125f;
    }
    // L = L0 F^-1, HIA = VT - L0 TX^T
    float L[3][3], HIA[3][4];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) L[r][c] = fmaf(L0[r][2], Fi[2][c], fmaf(L0[r][1], Fi[1][c], L0[r][0] * Fi[0][c]));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
            HIA[r][kk] = VT[r][kk] - fmaf(L0[r][2], TX[kk][2], fmaf(L0[r][1], TX[kk][1], L0[r][0] * TX[kk][0]));
    }
    const float vr = L[0][0] + L[1][1] + L[2][2];
    // Jaumann stress update
    float so[6], s[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) so[i] = S.sig[i * ss + si];
    // dt enters the increments as a float pair too: it changes little from
    // cycle to cycle, so its FP32 rounding would repeat with the same sign
    const float dt1_lo = static_cast<float>(dt1d - static_cast<double>(dt1));
    auto incr = [&](float g) { return fmaf(g, dt1, g * dt1_lo); };
    float eps[6] = {incr(L[0][0]), incr(L[1][1]), incr(L[2][2]), incr(0.5f * (L[0][1] + L[1][0])),
                    incr(0.5f * (L[0][2] + L[2][0])), incr(0.5f * (L[1][2] + L[2][1]))};
    {
        const float w0 = incr(0.5f * (L[0][1] - L[1][0]));
        const float w1 = incr(0.5f * (L[0][2] - L[2][0]));
        const float w2 = incr(0.5f * (L[1][2] - L[2][1]));
        const float tr = eps[0] + eps[1] + eps[2];
        // lambda and 2G enter as unevaluated pairs hi + lo of floats: a
        // stiffness rounded to FP32 is off by up to 6e-8 for every element
        // and cycle alike, which shifts all wave speeds and accumulates as
        // phase error; the pair carries the FP64 constants to ~1e-15
        const float lt = fmaf(lam_hi, tr, lam_lo * tr);
        float ge[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) ge[i] = fmaf(g2_hi, eps[i], g2_lo * eps[i]);
        s[0] = so[0] + lt + ge[0] + 2.f * so[3] * w0 + 2.f * so[4] * w1;
        s[1] = so[1] + lt + ge[1] - 2.f * so[3] * w0 + 2.f * so[5] * w2;
        s[2] = so[2] + lt + ge[2] - 2.f * so[4] * w1 - 2.f * so[5] * w2;
        s[3] = so[3] + ge[3] + (so[1] - so[0]) * w0 + so[5] * w1;
        s[4] = so[4] + ge[4] + (so[2] - so[0]) * w1 + so[5] * w0;
        s[5] = so[5] + ge[5] + (so[2] - so[1]) * w2 + so[3] * w1 - so[4] * w0;
    }
    if (PLASTIC) {
        const float pm = (s[0] + s[1] + s[2]) * (1.f / 3.f);
        const float d0 = s[0] - pm, d1 = s[1] - pm, d2 = s[2] - pm;
        const float j2 = 0.5f * (d0 * d0 + d1 * d1 + d2 * d2) + s[3] * s[3] + s[4] * s[4] + s[5] * s[5];
        const float seq = sqrtf(3.f * j2);
        const float ep_old = S.eps[si];
        const float sy = y0 + H * ep_old;
        if (seq > sy) {
            const float dl = (seq - sy) * M.mc.inv_3gh;
            const float r = 1.f - 3.f * G * dl / seq;
            s[0] = d0 * r + pm;
            s[1] = d1 * r + pm;
            s[2] = d2 * r + pm;
            s[3] *= r;
            s[4] *= r;
            s[5] *= r;
            if (!INIT) O.eps[oi] = ep_old + dl;
        }
    }
    if (!INIT) {
#pragma unroll
        for (int i = 0; i < 6; ++i) O.sig[i * os + oi] = s[i];
    }
    const float Vc = static_cast<float>(static_cast<double>(J) * S.vol0[si]);
    {
        float w = 0.f;
#pragma unroll
        for (int i = 0; i < 6; ++i) w += (i < 3 ? 0.5f : 1.0f) * (so[i] + s[i]) * eps[i];
        e_int += static_cast<double>(w * Vc);
    }
    const float DR = DRc * nx2 * Vc * dt1;
    const float cbe = S.cb[si];
    const float CR = CRc * invdet * (cbe * cbe);  // V0 / Vc = 1 / J
    float Gq[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const float h = fmaf(DR, HIA[i][kk], S.qia[(4 * i + kk) * ss + si]);
            if (!INIT) O.qia[(4 * i + kk) * os + oi] = h;
            Gq[i][kk] = fmaf(CR, HIA[i][kk], h);
        }
    const bool visc = !(fabsf(vr) < 1.0e-10f);
    float pv = 0.f;
    if (visc) {
        const float m0 = fminf(vr, 0.f);
        pv = rho * invdet * cbe * (cvisq * cvisq * cbe * vr * m0 - cvisl * wos * vr);
        e_vis += -static_cast<double>(pv * Vc * vr) * dt1d;
    }
    // Z = Vc F^-1 (sigma - p I) - W^T, W = Gq TX
    const float Sp[3][3] = {{s[0] - pv, s[3], s[4]}, {s[3], s[1] - pv, s[5]}, {s[4], s[5], s[2] - pv}};
    float W[3][3], Z[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            W[i][c] = fmaf(Gq[i][3], TX[3][c], fmaf(Gq[i][2], TX[2][c], fmaf(Gq[i][1], TX[1][c], Gq[i][0] * TX[0][c])));
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            Z[c][i] = Vc * fmaf(Fi[c][2], Sp[2][i], fmaf(Fi[c][1], Sp[1][i], Fi[c][0] * Sp[0][i])) - W[i][c];
    {
        // hourglass power sum_j h_j . v_j = Gq : HIA
        float hp = 0.f;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) hp = fmaf(Gq[i][kk], HIA[i][kk], hp);
        e_hg += static_cast<double>(hp) * dt1d;
    }
    // nodal forces f_j = -(B0_j Z) - Gamma_j Gq^T with B0_j Z = s_j^T Y / 8,
    // Y = A^T Z
    // (from a shared-memory stage, A and the connectivity are read again
    // here rather than kept in registers across the stress update)
    constexpr bool kReread = SMEM && ENSC_MIXED_REREAD;
    if (kReread) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                Ah[c][m] = S.a[(3 * c + m) * ss + si];
                Al[c][m] = S.a[(9 + 3 * c + m) * ss + si];
            }
    }
    float Y[3][3];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            float t = Al[0][m] * Z[0][i];
            t = fmaf(Al[1][m], Z[1][i], t);
            t = fmaf(Al[2][m], Z[2][i], t);
            t = fmaf(Ah[0][m], Z[0][i], t);
            t = fmaf(Ah[1][m], Z[1][i], t);
            t = fmaf(Ah[2][m], Z[2][i], t);
            Y[m][i] = 0.125f * t;
        }
    if (kReread) {
#pragma unroll
        for (int k = 0; k < 8; ++k) nk[k] = S.conn[k * ss + si];
    }
    // per force component: the node values of -(B0_j Z) - Gamma_j Gq^T from
    // their corner coefficients (-Y on xi, eta, zeta; -Gq on the hourglass
    // vectors, signed as Gamma)
    float f[3][8];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float c[8] = {0.f,          -Y[0][i],     -Y[1][i],     -Gq[i][0],
                      -Y[2][i],     Gq[i][2],     Gq[i][1],     -Gq[i][3]};
        corner_values(c, f[i]);
    }
    if (FOUT) {
#pragma unroll
        for (int i = 0; i < 24; ++i) fout[i] = f[i / 8][i % 8];
    } else {
        // (the force array is looked up here: a batch reads it from the stage)
        float* fe = static_cast<float*>(E.fe);
        auto store = [&](int j, int k, int64_t row, int64_t at) {
            *reinterpret_cast<float2*>(force_xy(fe, row, k, at)) = make_float2(f[0][j], f[1][j]);
            *force_z(fe, row, k, at) = f[2][j];
        };
        if (!E.slot_major) {
#pragma unroll
            for (int j = 0; j < 8; ++j) store(j, j, E.ne_pad, e);
        } else if (E.rows) {
            const uint32_t rows = __ldg(E.rows + e);
#pragma unroll
            for (int j = 0; j < 8; ++j) store(j, static_cast<int>((rows >> (4 * j)) & 7u), N.nn_pad, nk[j]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) store(j, j, N.nn_pad, nk[j]);
        }
    }
    // element dt (compute_dtStable, exDyna3D.cpp:828-834), with the
    // divisions by wos as products with its reciprocal
    {
        const double m0 = fmin(static_cast<double>(vr), 0.0);
        const double xi = M.cvisl - M.mc.cq2_wos * len * m0;
        dts = (sqrt(1.0 + xi * xi) - xi) * len * M.mc.inv_wos;
    }
    if (!isfinite(dts)) bad |= ST_NONFINITE;
}

// The init force pass (dt = 0, no state written, no energy), from the tiles
// in global memory.
template <bool PLASTIC>
__global__ void __launch_bounds__(kElemThreads, ENSC_ELEM_MINB_MIXED)
    k_element_mixed_init(ElemArrays E, NodeArrays N, Material M, Ctl* ctl) {
    if (ctl->done) return;
    const int64_t ne = E.ne;
    double e_int = 0.0, e_hg = 0.0, e_vis = 0.0;
    double dts_min = DBL_MAX, len_min = DBL_MAX;
    int32_t bad = 0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < ne; e += stride) {
        unsigned char* g = mixed_tile(E, e >> 5);
        const int lane = static_cast<int>(e & 31);
        double dts, len;
        element_body_mixed<PLASTIC, true>(E, N, M, mixed_src_tile(g, lane), mixed_out_tile(g, lane), 0.f, 0.0, e, dts, len,
                                          e_int, e_hg, e_vis, bad);
        dts_min = fmin(dts_min, dts);
        len_min = fmin(len_min, len);
    }
    if (bad) atomicOr(&ctl->status, bad);
    block_min2_d<kElemThreads>(dts_min, len_min, &ctl->dts_next, &ctl->len_min);
}

// ---- warp-pipelined element pass -----------------------------------------
// Every warp runs its own pipeline over tiles of 32 consecutive elements: two
// shared-memory stages, each filled by one bulk copy of a whole tile while
// the other is computed, and no block-wide barrier per tile.  Node data are
// gathered from global memory, and all outputs are written there.
constexpr int kMixedPipeWarps = ENSC_MIXED_PIPE_WARPS;
constexpr size_t kMixedPipeSmem = static_cast<size_t>(kMixedPipeWarps) * (2 * MixedTile::kBytes + 16);

// Lane 0: the tile at src into shared memory at dst, completing on bar
// (elastic instances leave out eps_p, the tile's last row).
template <bool PLASTIC>
__device__ __forceinline__ void mixed_tile_issue(const void* src, uint32_t dst, uint32_t bar) {
    constexpr uint32_t bytes = PLASTIC ? MixedTile::kBytes : MixedTile::kEps;
    mbar_arrive_expect_tx(bar, bytes);
    fence_proxy_async_smem();  // the warp's reads of this stage come before the copy into it
    bulk_g2s(dst, src, bytes, bar);
}

template <bool PLASTIC>
__global__ void __launch_bounds__(32 * kMixedPipeWarps, ENSC_MIXED_PIPE_MINB)
    k_element_mixed_warp(ElemArrays E, NodeArrays N, Material M, Ctl* ctl, Partials P) {
    constexpr uint32_t SB = MixedTile::kBytes;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    unsigned char* wst = smem + static_cast<size_t>(wid) * 2 * SB;
    const uint32_t stage0 = smem_addr(wst);
    const uint32_t bar0 = smem_addr(smem + static_cast<size_t>(kMixedPipeWarps) * 2 * SB) + 16u * wid;
    const int ntiles = static_cast<int>((E.ne + 31) / 32);
    const int wstride = static_cast<int>(gridDim.x) * kMixedPipeWarps;
    const int w0 = static_cast<int>(blockIdx.x) * kMixedPipeWarps + wid;
    if (lane == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
        for (int s = 0; s < 2; ++s) {
            const int t = w0 + s * wstride;
            if (t < ntiles) mixed_tile_issue<PLASTIC>(mixed_tile(E, t), stage0 + s * SB, bar0 + 8 * s);
        }
    }
    __syncwarp();
    cycle_kernel_enter();  // (the last element pass completed before the kernel before this one began)
    if (ctl->done) {
        for (int s = 0; s < 2; ++s)
            if (w0 + s * wstride < ntiles) mbar_wait_bounded(bar0 + 8 * s, 0);
        return;
    }
    const double dt1d = ctl->dt_i_1;
    const float dt1 = static_cast<float>(dt1d);
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
            double dts, len;
            element_body_mixed<PLASTIC, false, true>(
                E, N, M, mixed_src_tile(wst + s * SB, lane), mixed_out_tile(mixed_tile(E, t), lane), dt1, dt1d, e, dts,
                len, e_int, e_hg, e_vis, bad);
            dts_min = fmin(dts_min, dts);
            len_min = fmin(len_min, len);
        }
        __syncwarp();  // all lanes are done with stage s
        const int tn = t + 2 * wstride;
        if (lane == 0 && tn < ntiles) mixed_tile_issue<PLASTIC>(mixed_tile(E, tn), stage0 + s * SB, bar);
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
    block_min2_d<32 * kMixedPipeWarps>(dts_min, len_min, &ctl->dts_next, &ctl->len_min);
    double v3[3] = {e_int, e_hg, e_vis};
    block_sum_d<32 * kMixedPipeWarps, 3, 7u>(v3, P.elem, P.n_elem_blocks, blockIdx.x);
}

// ---- element pass with patch assembly -------------------------------------
// One patch, two consecutive tiles, per 64-thread block at a time, through two
// stages.  After its element body a thread holds its element's 24 nodal
// forces; once the whole block is done with the stage's inputs, the forces go
// into the stage's memory as [3][8 slots][kPatchElems elements], and the block
// sums each of the patch's nodes over its incidences in slot order (starting
// from zero) and writes the node's partial to PA.pf.  INIT: the init force pass
// (dt = 0, no state written, no energy).
constexpr uint32_t kPatchTiles = kPatchElems / 32;
constexpr uint32_t kPatchStageBytes = kPatchTiles * MixedTile::kBytes;
constexpr size_t kPatchSmem = 2 * static_cast<size_t>(kPatchStageBytes) + 16;
static_assert(3u * 8u * kPatchElems * 4u <= kPatchStageBytes, "the element forces fit in a stage");

__device__ __forceinline__ void patch_partials(const PatchArrays& E, const float* sf, int64_t t, int tid) {
    const uint32_t q0 = __ldg(E.pf_off + t), q1 = __ldg(E.pf_off + t + 1);
    for (uint32_t q = q0 + tid; q < q1; q += kPatchElems) {
        const uint32_t a = __ldg(E.pinc_off + q), b = __ldg(E.pinc_off + q + 1);
        float f0 = 0.f, f1 = 0.f, f2 = 0.f;
        for (uint32_t r = a; r < b; ++r) {
            const uint32_t u = __ldg(E.pinc + r);
            const uint32_t col = (u & 7u) * kPatchElems + (u >> 3);
            f0 += sf[col];
            f1 += sf[8 * kPatchElems + col];
            f2 += sf[16 * kPatchElems + col];
        }
        E.pf[q] = f0;
        E.pf[E.pf_pad + q] = f1;
        E.pf[2 * E.pf_pad + q] = f2;
    }
}

template <bool PLASTIC, bool INIT>
__global__ void __launch_bounds__(kPatchElems, 8)
    k_element_mixed_patch(ElemArrays E, NodeArrays N, Material M, Ctl* ctl, Partials P, PatchArrays PA) {
    cycle_kernel_enter();
    if (ctl->done) return;
    extern __shared__ __align__(128) unsigned char smem[];
    const float dt1 = INIT ? 0.f : static_cast<float>(ctl->dt_i_1);
    const double dt1d = INIT ? 0.0 : ctl->dt_i_1;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t stage0 = smem_addr(smem);
    const uint32_t bar0 = stage0 + 2 * kPatchStageBytes;
    const int64_t ntiles = (E.ne + 31) / 32, npatch = (E.ne + kPatchElems - 1) / kPatchElems;
    const int64_t gstride = gridDim.x;
    auto issue = [&](int64_t p, int s) {
        const int64_t left = ntiles - p * kPatchTiles;
        const uint32_t bytes = static_cast<uint32_t>(left < kPatchTiles ? left : kPatchTiles) * MixedTile::kBytes;
        mbar_arrive_expect_tx(bar0 + 8 * s, bytes);
        fence_proxy_async_smem();  // the block's reads of this stage come before the copy into it
        bulk_g2s(stage0 + s * kPatchStageBytes, mixed_tile(E, p * kPatchTiles), bytes, bar0 + 8 * s);
    };
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
        for (int s = 0; s < 2; ++s)
            if (blockIdx.x + s * gstride < npatch) issue(blockIdx.x + s * gstride, s);
    }
    __syncthreads();
    double e_int = 0.0, e_hg = 0.0, e_vis = 0.0;
    double dts_min = DBL_MAX, len_min = DBL_MAX;
    int32_t bad = 0;
    bool timed_out = false;
    int it = 0;
    for (int64_t t = blockIdx.x; t < npatch; t += gstride, ++it) {
        const int s = it & 1;
        const bool ok = mbar_wait_bounded(bar0 + 8 * s, (it >> 1) & 1);
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        unsigned char* st = smem + s * kPatchStageBytes;
        const int64_t e = t * kPatchElems + tid;
        const bool live = e < E.ne;
        float fo[24];
        if (live) {
            double dts, len;
            element_body_mixed<PLASTIC, INIT, true, true>(
                E, N, M, mixed_src_tile(st + wid * MixedTile::kBytes, lane),
                mixed_out_tile(mixed_tile(E, t * kPatchTiles + wid), lane), dt1, dt1d, e, dts, len, e_int, e_hg, e_vis, bad,
                fo);
            dts_min = fmin(dts_min, dts);
            len_min = fmin(len_min, len);
        }
        __syncthreads();  // the stage's inputs are consumed
        float* sf = reinterpret_cast<float*>(st);
        if (live) {
#pragma unroll
            for (int i = 0; i < 24; ++i) sf[i * kPatchElems + tid] = fo[i];
        }
        __syncthreads();
        patch_partials(PA, sf, t, tid);
        __syncthreads();  // the block is done with stage s
        const int64_t tn = t + 2 * gstride;
        if (tid == 0 && tn < npatch) issue(tn, s);
    }
    if (timed_out) {
        if (tid == 0) {
            atomicOr(&ctl->status, ST_TIMEOUT);
            for (int k = 0; k < 2; ++k) {
                const int itk = it + k;
                if (blockIdx.x + itk * gstride < npatch) mbar_wait_bounded(bar0 + 8 * (itk & 1), (itk >> 1) & 1);
            }
        }
        __syncthreads();
    }
    if (bad) atomicOr(&ctl->status, bad);
    block_min2_d<kPatchElems>(dts_min, len_min, &ctl->dts_next, &ctl->len_min);
    if (!INIT) {
        double v3[3] = {e_int, e_hg, e_vis};
        block_sum_d<kPatchElems, 3, 7u>(v3, P.elem, P.n_elem_blocks, blockIdx.x);
    }
}

// One node's force under the patch assembly: its partials in patch order,
// from zero.
__device__ __forceinline__ void patch_gather(const PatchArrays& PA, int64_t n, float (&f)[3]) {
    const int64_t pp = PA.pf_pad;
    for (uint32_t r = __ldg(PA.nptr + n), b = __ldg(PA.nptr + n + 1); r < b; ++r) {
        const uint32_t q = __ldg(PA.nent + r);
        f[0] += __ldg(PA.pf + q);
        f[1] += __ldg(PA.pf + pp + q);
        f[2] += __ldg(PA.pf + 2 * pp + q);
    }
}

// The velocity update in FP64 on the split velocity (hi float + 16-bit
// residual, v_join / v_split): v + (dt_i + dt_i_1) / 2 * a with the FP32
// acceleration a = f M^-1 (inverse mass as a float pair); returns the new
// velocity as a double and its split form.
__device__ __forceinline__ double velocity_update_split(double vo, float f, double im, double hdt, float& hi,
                                                        int16_t& lo) {
    const float im_hi = static_cast<float>(im);
    const float im_lo = static_cast<float>(im - static_cast<double>(im_hi));
    const float acc = fmaf(f, im_hi, f * im_lo);
    const double vn = fma(hdt, static_cast<double>(acc), vo);
    v_split(vn, hi, lo);
    return vn;
}

// The force of one node from per-element forces, through the general lists
// (meshes whose nodes repeat slots).
__device__ __forceinline__ void listed_forces_mixed(const ElemArrays& E, const NodeArrays& N, const int64_t n,
                                                    float (&f)[3]) {
    const float* fe = static_cast<const float*>(E.fe);
    f[0] = f[1] = f[2] = 0.f;
    for (int64_t i = N.csr_ptr[n]; i < N.csr_ptr[n + 1]; ++i) {
        const uint32_t ent = N.csr_ent[i];
        const int k = static_cast<int>(ent & 7u);
        const uint32_t el = ent >> 3;
        const float2 xy = *reinterpret_cast<const float2*>(force_xy(fe, E.ne_pad, k, el));
        f[0] += xy.x;
        f[1] += xy.y;
        f[2] += *force_z(fe, E.ne_pad, k, el);
    }
}

// The work of a node update: all of it; all but the kinetic energy (a resident run
// in every cycle); or the kinetic energy of the velocities that the update will
// form and nothing else (a resident run ahead of its last update).
enum NodeWork { kNodeAll, kNodeUpdate, kNodeKinetic };

// One node of the mixed node pass where the forces are per element; shared by
// the single-instance, batched and resident-run kernels.
template <NodeWork WORK = kNodeAll>
__device__ __forceinline__ void node_body_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M,
                                                const double dt_i, const double dt_i_1, const double amp, const int64_t n,
                                                double& kin, double& wext, int32_t& bad) {
    const int64_t np = N.nn_pad;
    const double dt_avg = 0.5 * (dt_i + dt_i_1);
    float f[3];
    listed_forces_mixed(E, N, n, f);
    const double im = N.inv_mass[n];
    const uint32_t code = N.bc[n];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float a = f[c];
        float g = 0.f;
        if (M.gravity_on) {
            g = static_cast<float>(amp * M.gravity_value * M.gravity_dir[c] / im);
            a += g;
        }
        const uint32_t cc = (code >> (2 * c)) & 3u;
        float r = 0.f, rf = 0.f;
        if (cc & 2u) {
            r = -a;
            a = 0.f;
        }
        if ((cc & 1u) && a != 0.f) {
            rf = -a;
            r = -a;
            a = 0.f;
        }
        if (WORK != kNodeKinetic && cc) N.rf[c * np + n] = static_cast<double>(rf);
        float* pv = node_vf(N, c, n);
        int16_t* pl = v_lo_rows(N.v, np) + c * np + n;
        double* px = node_x(N, c, n);
        const double vod = v_join(*pv, *pl);
        float vn;
        int16_t vl;
        const double vnd = velocity_update_split(vod, a, im, dt_avg, vn, vl);
        if (WORK != kNodeKinetic) {
            *pv = vn;
            *pl = vl;
            *px += dt_i * vnd;
            wext += static_cast<double>(g + r) * dt_avg * 0.5 * (vod + vnd);
        }
        if (WORK != kNodeUpdate) kin += 0.5 * (vnd * vnd) / im;
        if (WORK != kNodeKinetic && !isfinite(vnd)) bad |= ST_NONFINITE;
    }
}

// W consecutive nodes of the mixed node pass; per node the arithmetic of
// node_body_mixed.  Every slot is added, empty ones as the zeros they hold: the
// slot-major rows start zeroed and only the slot's element writes them.  Nodes
// at or past nn (row padding) are loaded and stored back unchanged.
//
// pre (resident runs): the nodes' own records, loaded while the grid still works
// on the forces.
template <int W>
struct NodeRowsMixed {
    double im[W], q[W][4];
    float vz[W];
    int16_t lo[3][W];
    uint32_t code;
};
template <int W>
__device__ __forceinline__ void node_rows_load(const NodeView& N, const int64_t n0, NodeRowsMixed<W>& r) {
#pragma unroll
    for (int j = 0; j < W; ++j) ld_rec(N.x + 4 * (n0 + j), r.q[j]);
    ld_row<W>(static_cast<const float*>(N.v) + n0, r.vz);
#pragma unroll
    for (int c = 0; c < 3; ++c) ld_row<W>(v_lo_rows(N.v, N.np) + c * N.np + n0, r.lo[c]);
    ld_row<W>(N.inv_mass + n0, r.im);
    r.code = ld_bytes<W>(N.bc + n0);
}

// The forces of W consecutive nodes: their slots in order, or their patch
// partials in patch order.
template <int W, bool PATCH>
__device__ __forceinline__ void node_forces_mixed(const NodeView& N, const int64_t n0, float (&f)[3][W]) {
    const int64_t np = N.np;
    const float* fe = static_cast<const float*>(N.fe);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int j = 0; j < W; ++j) f[c][j] = 0.f;
    if constexpr (PATCH) {
        // patch assembly: the node's partials in patch order
        uint32_t lo[W], bnd[W + 1];
        ld_row<W>(N.nptr + n0, lo);
#pragma unroll
        for (int j = 0; j < W; ++j) bnd[j] = lo[j];
        bnd[W] = __ldg(N.nptr + n0 + W);
        const int64_t pp = N.pf_pad;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            for (uint32_t r = bnd[j]; r < bnd[j + 1]; ++r) {
                const uint32_t q = __ldg(N.nent + r);
                f[0][j] += __ldg(N.pf + q);
                f[1][j] += __ldg(N.pf + pp + q);
                f[2][j] += __ldg(N.pf + 2 * pp + q);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float xy[2 * W], z[W];
            ld_row<2 * W>(force_xy(fe, np, k, n0), xy);
            ld_row<W>(force_z(fe, np, k, n0), z);
#pragma unroll
            for (int j = 0; j < W; ++j) {
                f[0][j] += xy[2 * j];
                f[1][j] += xy[2 * j + 1];
                f[2][j] += z[j];
            }
        }
    }
}

// PRE: rows and forces come in pre and fpre.
template <int W, bool PATCH, bool PRE = false, NodeWork WORK = kNodeAll>
__device__ __forceinline__ void node_group_mixed(const NodeView& N, const double dt_i, const double dt_i_1,
                                                 const double amp, const int64_t n0, double& kin, double& wext,
                                                 int32_t& bad, const NodeRowsMixed<W>* pre = nullptr,
                                                 const float (*fpre)[W] = nullptr) {
    const int64_t np = N.np, nn = N.nn;
    const double dt_avg = 0.5 * (dt_i + dt_i_1);
    // the nodes' own rows first, so that their loads are in flight with the
    // force slots'
    NodeRowsMixed<W> own;
    if constexpr (PRE) own = *pre;
    else node_rows_load<W>(N, n0, own);
    float f[3][W];
    if constexpr (PRE) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int j = 0; j < W; ++j) f[c][j] = fpre[c][j];
    } else {
        node_forces_mixed<W, PATCH>(N, n0, f);
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (n0 + j >= nn) continue;
        const double im = own.im[j];
        float v[3] = {rec_vx(own.q[j][3]), rec_vy(own.q[j][3]), own.vz[j]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float a = f[c][j];
            float g = 0.f;
            if (N.gravity_on) {
                g = static_cast<float>(amp * N.gravity_value * N.gravity_dir[c] / im);
                a += g;
            }
            const uint32_t cc = (own.code >> (8 * j + 2 * c)) & 3u;
            float r = 0.f, rf = 0.f;
            if (cc & 2u) {
                r = -a;
                a = 0.f;
            }
            if ((cc & 1u) && a != 0.f) {
                rf = -a;
                r = -a;
                a = 0.f;
            }
            if (WORK != kNodeKinetic && cc) N.rf[c * np + n0 + j] = static_cast<double>(rf);
            const double vod = v_join(v[c], own.lo[c][j]);
            const double vnd = velocity_update_split(vod, a, im, dt_avg, v[c], own.lo[c][j]);
            if (WORK != kNodeKinetic) {
                own.q[j][c] = own.q[j][c] + dt_i * vnd;
                wext += static_cast<double>(g + r) * dt_avg * 0.5 * (vod + vnd);
            }
            if (WORK != kNodeUpdate) kin += 0.5 * (vnd * vnd) / im;
            if (WORK != kNodeKinetic && !isfinite(vnd)) bad |= ST_NONFINITE;
        }
        own.q[j][3] = rec_vxy(v[0], v[1]);
        own.vz[j] = v[2];
    }
    if (WORK == kNodeKinetic) return;
#pragma unroll
    for (int j = 0; j < W; ++j) st_rec(N.x + 4 * (n0 + j), own.q[j]);
    st_row<W>(static_cast<float*>(N.v) + n0, own.vz);
#pragma unroll
    for (int c = 0; c < 3; ++c) st_row<W>(v_lo_rows(N.v, np) + c * np + n0, own.lo[c]);
}

// Node pass in mixed precision: FP32 slot-ordered gather and acceleration,
// FP32 velocity, FP64 position accumulation and energy (the u rows hold the
// reference position x - u and are not touched).
// PATCH: the instance uses the patch assembly (one instantiation each, so
// the slot-assembly pass carries no code of the other).
template <bool PATCH>
__global__ void __launch_bounds__(kNodeThreads, ENSC_NODE_MINB_MIXED) k_node_mixed(ElemArrays E, NodeArrays N, Material M, Ctl* ctl,
                                                             Partials P, PatchArrays PA) {
    cycle_kernel_enter();
    if (ctl->done) return;
    double dt_i;
    const double dt_i_1 = ctl->dt_i_1;
    if (ctl->dt_final) {
        dt_i = ctl->dt_i;
    } else {
        double d = bits_ord(ctl->len_min) / ctl->wos;
        d = d < ctl->dts_cur ? d : ctl->dts_cur;
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
        constexpr int W = kNodeGroupMixed;
        const NodeView nv = node_view(E, N, M, ctl, &PA);
        // from the last nodes back: their forces are the latest in L2, and the
        // first nodes' records stay there for the next element pass (B200,
        // 2,097,152 elements: 3% of a mixed cycle, 2% of an FP64 one)
        const int64_t ng = (nn + W - 1) / W;
        for (int64_t g = t0; g < ng; g += stride)
            node_group_mixed<W, PATCH>(nv, dt_i, dt_i_1, amp, (ng - 1 - g) * W, kin, wext, bad);
    } else {
        for (int64_t n = t0; n < nn; n += stride) node_body_mixed(E, N, M, dt_i, dt_i_1, amp, n, kin, wext, bad);
    }
    if (bad) atomicOr(&ctl->status, bad);
    double v2[2] = {kin, wext};
    block_sum_d<kNodeThreads, 2, 2u>(v2, P.node, P.n_node_blocks, blockIdx.x);
}

// ---- resident runs (ensc_run.cuh) -----------------------------------------
// 16 warps per SM as in the warp-pipelined pass; a tile takes 6,144 bytes, so
// that 37 tiles fit an SM and 148 SMs hold 151,552 elements at two tiles per
// warp.
constexpr int kRunWarpsMixed = 16;
template <bool PLASTIC>
struct RunMixed {
    static constexpr uint32_t kTileBytes = MixedTile::kBytes;
    static constexpr bool kKinInUpdate = true;
    __device__ static const uint32_t* conn(const unsigned char* tile) {
        return reinterpret_cast<const uint32_t*>(tile);
    }
    __device__ static void load_tile(const ElemArrays& E, uint32_t dst, uint32_t bar, int64_t t, int lane) {
        if (lane == 0) mixed_tile_issue<PLASTIC>(mixed_tile(E, t), dst, bar);
    }
    __device__ static void store_tile(const ElemArrays& E, const unsigned char* tile, int64_t t, int lane) {
        // whole rows: the entries past ne are padding
        unsigned char* g = mixed_tile(E, t);
        constexpr uint32_t end = PLASTIC ? MixedTile::kBytes : MixedTile::kEps;
        for (uint32_t o = MixedTile::kState + 4u * lane; o < end; o += 128)
            *reinterpret_cast<float*>(g + o) = *reinterpret_cast<const float*>(tile + o);
    }
    __device__ static void element(const ElemArrays& E, const NodeArrays& N, const Material& M, unsigned char* tile,
                                   double dt1, int64_t e, int lane, double& dts, double& len, double& e_int,
                                   double& e_hg, double& e_vis, int32_t& bad) {
        element_body_mixed<PLASTIC, false, true>(E, N, M, mixed_src_tile(tile, lane),
                                                                      mixed_out_tile(tile, lane),
                                                                      static_cast<float>(dt1), dt1, e, dts, len, e_int,
                                                                      e_hg, e_vis, bad);
    }
    // as RunFp64::Nodes
    template <int W>
    struct Nodes {
        NodeRowsMixed<W> rows;
        float f[3][W];
        __device__ void load(const ElemArrays& E, const NodeArrays& N, const Material& M, int64_t t0) {
            if (E.slot_major && t0 * W < N.nn) node_rows_load<W>(node_view(E, N, M, nullptr), t0 * W, rows);
        }
        __device__ void gather(const ElemArrays& E, const NodeArrays& N, const Material& M, int64_t t0) {
            if (E.slot_major && t0 * W < N.nn) node_forces_mixed<W, false>(node_view(E, N, M, nullptr), t0 * W, f);
        }
        template <NodeWork WORK>
        __device__ void pass(const ElemArrays& E, const NodeArrays& N, const Material& M, double dt_i, double dt_i_1,
                             double amp, int64_t t0, int64_t stride, double& kin, double& wext, int32_t& bad) {
            if (E.slot_major) {
                const NodeView nv = node_view(E, N, M, nullptr);
                if (t0 * W < N.nn)
                    node_group_mixed<W, false, true, WORK>(nv, dt_i, dt_i_1, amp, t0 * W, kin, wext, bad, &rows, f);
                if (W > 1)
                    for (int64_t g = t0 + stride; g * W < N.nn; g += stride) {
                        NodeRowsMixed<W> r;
                        float fg[3][W];
                        node_rows_load<W>(nv, g * W, r);
                        node_forces_mixed<W, false>(nv, g * W, fg);
                        node_group_mixed<W, false, true, WORK>(nv, dt_i, dt_i_1, amp, g * W, kin, wext, bad, &r, fg);
                    }
            } else {
                for (int64_t n = t0; n < N.nn; n += stride)
                    node_body_mixed<WORK>(E, N, M, dt_i, dt_i_1, amp, n, kin, wext, bad);
            }
        }
        __device__ void update(const ElemArrays& E, const NodeArrays& N, const Material& M, double dt_i, double dt_i_1,
                               double amp, int64_t t0, int64_t stride, double& wext, int32_t& bad) {
            double kin = 0.0;
            pass<kNodeUpdate>(E, N, M, dt_i, dt_i_1, amp, t0, stride, kin, wext, bad);
        }
        // the kinetic energy of the velocities that the update will form
        __device__ double kinetic_after(const ElemArrays& E, const NodeArrays& N, const Material& M, double dt_i,
                                        double dt_i_1, double amp, int64_t t0, int64_t stride) {
            double kin = 0.0, wext = 0.0;
            int32_t bad = 0;
            pass<kNodeKinetic>(E, N, M, dt_i, dt_i_1, amp, t0, stride, kin, wext, bad);
            return kin;
        }
    };
    __device__ static double kinetic(const NodeArrays& N, int64_t n) {
        double kin = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double v = v_join(*node_vf(N, c, n), v_lo_rows(N.v, N.nn_pad)[c * N.nn_pad + n]);
            kin += 0.5 * (v * v) / N.inv_mass[n];
        }
        return kin;
    }
};

template <bool PLASTIC, bool CLUSTER, int W>
__global__ void __launch_bounds__(CLUSTER ? 128 : 32 * kRunWarpsMixed, 1)
    k_run_mixed(ElemArrays E, NodeArrays N, Material M, Ctl* ctl, Partials P, RunSync* sync, RunArgs a) {
    run_cycles<RunMixed<PLASTIC>, CLUSTER, W>(E, N, M, ctl, P, sync, a);
}

// The last cycle's acceleration in mixed precision (see k_acceleration in
// the FP64 stepper): the FP32 force sum, gravity and the FP32 acceleration
// f M^-1 that the mixed node pass feeds into the velocity update, written
// as doubles, interleaved xyz per node.
__global__ void __launch_bounds__(kNodeThreads) k_acceleration_mixed(PatchArrays PA, ElemArrays E, NodeArrays N, Material M,
                                                                     const Ctl* ctl, double* a_out) {
    const double amp = (M.gravity_on && M.amp_n > 0) ? gravity_amplitude(M.amp, M.amp_n, ctl->time, ctl->dt_i) : 1.0;
    const NodeView nv = node_view(E, N, M, nullptr, &PA);
    for (int64_t n = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; n < N.nn;
         n += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        float f[3] = {0.f, 0.f, 0.f};
        if (PA.pf) {
            patch_gather(PA, n, f);
        } else if (E.slot_major) {
            float g[3][1];
            node_forces_mixed<1, false>(nv, n, g);
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] = g[c][0];
        } else {
            listed_forces_mixed(E, N, n, f);
        }
        const double im = N.inv_mass[n];
        const float im_hi = static_cast<float>(im);
        const float im_lo = static_cast<float>(im - static_cast<double>(im_hi));
        const uint32_t code = N.bc[n];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float a = f[c];
            if (M.gravity_on) a += static_cast<float>(amp * M.gravity_value * M.gravity_dir[c] / im);
            const uint32_t cc = (code >> (2 * c)) & 3u;
            if (cc & 2u) a = 0.f;
            if ((cc & 1u) && a != 0.f) a = 0.f;
            a_out[3 * n + c] = static_cast<double>(fmaf(a, im_hi, a * im_lo));
        }
    }
}

// ---- batched instances --------------------------------------------------------
// Element tiles of 32 elements (under the patch assembly: patches, two tiles)
// and node tiles of 32 * kNodeGroupBatchMixed nodes, each inside one instance
// whose arrays, material and control block come from the instance table.  The
// element pass runs one pipeline per warp over the tile list (one per block
// over patches); the node pass gives each node tile to one warp.  Each tile
// accumulates its work terms across cycles (one owner per tile and pass) and
// keeps its latest kinetic energy; k_fold_batch folds them per instance in tile
// order, so the totals do not depend on scheduling.
// A batch stage: the tile (or patch), then its instance descriptor, its
// element-pass scalars (StageHdr), the TileInfo the filling lane writes, and the
// ETileSrc record of the tile that uses the stage next.  Every tile is copied
// whole whether or not its instance runs this cycle; the consumer skips the
// tiles of instances that do not.  One lane fills a stage.
template <uint32_t ROOM>
__device__ __forceinline__ void batch_issue(const BatchTables& T, const ETileSrc& src, int64_t t_next, int64_t ntiles,
                                            unsigned char* stage, uint32_t dst, uint32_t bar) {
    const bool next = t_next < ntiles;
    TileInfo* ti = reinterpret_cast<TileInfo*>(stage + ROOM + kBatchInfoOff);
    ti->slot = src.slot;
    ti->base = src.base;
    mbar_arrive_expect_tx(bar, static_cast<uint32_t>(src.bytes) + sizeof(InstanceDesc) + sizeof(StageHdr) +
                                   (next ? sizeof(ETileSrc) : 0u));
    fence_proxy_async_smem();  // the reads of this stage come before the copies into it
    bulk_g2s(dst, src.tile, static_cast<uint32_t>(src.bytes), bar);
    bulk_g2s(dst + ROOM, T.desc + src.slot, sizeof(InstanceDesc), bar);
    bulk_g2s(dst + ROOM + kBatchHdrOff, T.sparam + src.slot, sizeof(StageHdr), bar);
    if (next) bulk_g2s(dst + ROOM + kBatchNextOff, T.etile_src + t_next, sizeof(ETileSrc), bar);
}

constexpr uint32_t kBatchStageMixed = MixedTile::kBytes + kBatchTailBytes;
constexpr size_t kBatchMixedSmem = static_cast<size_t>(kMixedPipeWarps) * (2 * kBatchStageMixed + 16);

__global__ void __launch_bounds__(32 * kMixedPipeWarps, ENSC_MIXED_PIPE_MINB) k_element_batch_mixed(BatchTables T) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr uint32_t SB = kBatchStageMixed;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    unsigned char* wst = smem + static_cast<size_t>(wid) * 2 * SB;
    const uint32_t stage0 = smem_addr(wst);
    const uint32_t bar0 = smem_addr(smem + static_cast<size_t>(kMixedPipeWarps) * 2 * SB) + 16u * wid;
    __shared__ SentMinima sent[kMixedPipeWarps];
    if (lane == 0) sent[wid].slot = -1;
    cycle_kernel_enter();
    const int ntiles = T.counts[0];
    const int wstride = static_cast<int>(gridDim.x) * kMixedPipeWarps;
    const int w0 = static_cast<int>(blockIdx.x) * kMixedPipeWarps + wid;
    if (lane == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
        for (int s = 0; s < 2; ++s) {
            const int t = w0 + s * wstride;
            if (t < ntiles)
                batch_issue<MixedTile::kBytes>(T, T.etile_src[t], t + 2 * wstride, ntiles, wst + s * SB, stage0 + s * SB,
                                               bar0 + 8 * s);
        }
    }
    __syncwarp();
    bool timed_out = false;
    int it = 0;
    int t = w0;
    for (; t < ntiles; t += wstride, ++it) {
        const int s = it & 1;
        const uint32_t bar = bar0 + 8 * s;
        const bool ok = mbar_wait_bounded(bar, (it >> 1) & 1);
        if (__any_sync(0xffffffffu, !ok)) {
            timed_out = true;
            break;
        }
        unsigned char* sb = wst + s * SB;
        unsigned char* tail = sb + MixedTile::kBytes;
        const InstanceDesc& d = *reinterpret_cast<const InstanceDesc*>(tail);
        const StageHdr& h = *reinterpret_cast<const StageHdr*>(tail + kBatchHdrOff);
        const TileInfo& ti = *reinterpret_cast<const TileInfo*>(tail + kBatchInfoOff);
        double ei = 0.0, eh = 0.0, ev = 0.0, dts = DBL_MAX, len = DBL_MAX;
        int32_t bad = 0;
        const int slot = ti.slot, e = ti.base + lane;
        const bool live = h.live != 0;
        if (live && e < d.E.ne) {
            const ElemArrays& E = d.E;
            const NodeArrays& N = d.N;
            const double dt1d = h.dt1;
            element_body_mixed<true, false, true>(
                E, N, d.M, mixed_src_tile(sb, lane), mixed_out_tile(mixed_tile(E, ti.base >> 5), lane),
                static_cast<float>(dt1d), dt1d, e, dts, len, ei, eh, ev, bad);
        }
        __syncwarp();  // all lanes are done with stage s
        const int tn = t + 2 * wstride;
        if (lane == 0 && tn < ntiles) {
            const ETileSrc src = *reinterpret_cast<const ETileSrc*>(tail + kBatchNextOff);
            batch_issue<MixedTile::kBytes>(T, src, tn + 2 * wstride, ntiles, sb, stage0 + s * SB, bar);
        }
        if (live) batch_tile_sums(T, t, slot, lane, ei, eh, ev, dts, len, bad, &sent[wid]);
    }
    if (timed_out && lane == 0) {
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

// The same under the patch assembly (a batch has one assembly): one patch per
// block at a time, as k_element_mixed_patch.
constexpr uint32_t kBatchStagePatch = kPatchStageBytes + kBatchTailBytes;
constexpr size_t kBatchPatchSmem = 2 * static_cast<size_t>(kBatchStagePatch) + 16;

__global__ void __launch_bounds__(kPatchElems, 8) k_element_batch_patch(BatchTables T) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr uint32_t SB = kBatchStagePatch;
    constexpr int NW = kPatchElems / 32;  // energy partial slots per patch
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t stage0 = smem_addr(smem);
    const uint32_t bar0 = stage0 + 2 * SB;
    __shared__ SentMinima sent[kPatchElems / 32];
    if (lane == 0) sent[wid].slot = -1;
    cycle_kernel_enter();
    const int64_t ntiles = T.counts[0];
    const int64_t gstride = gridDim.x;
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
        for (int s = 0; s < 2; ++s) {
            const int64_t t = blockIdx.x + s * gstride;
            if (t < ntiles)
                batch_issue<kPatchStageBytes>(T, T.etile_src[t], t + 2 * gstride, ntiles, smem + s * SB, stage0 + s * SB,
                                              bar0 + 8 * s);
        }
    }
    __syncthreads();
    bool timed_out = false;
    int it = 0;
    int64_t t = blockIdx.x;
    for (; t < ntiles; t += gstride, ++it) {
        const int s = it & 1;
        const uint32_t bar = bar0 + 8 * s;
        const bool ok = mbar_wait_bounded(bar, (it >> 1) & 1);
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        unsigned char* sb = smem + s * SB;
        unsigned char* tail = sb + kPatchStageBytes;
        const InstanceDesc& d = *reinterpret_cast<const InstanceDesc*>(tail);
        const StageHdr& h = *reinterpret_cast<const StageHdr*>(tail + kBatchHdrOff);
        const TileInfo& ti = *reinterpret_cast<const TileInfo*>(tail + kBatchInfoOff);
        double ei = 0.0, eh = 0.0, ev = 0.0, dts = DBL_MAX, len = DBL_MAX;
        int32_t bad = 0;
        const int slot = ti.slot;
        const bool live = h.live != 0;
        float fo[24];
        const int64_t e = static_cast<int64_t>(ti.base) + tid;
        const int64_t ne = d.E.ne;
        if (live && e < ne) {
            const ElemArrays& E = d.E;
            const NodeArrays& N = d.N;
            const double dt1d = h.dt1;
            element_body_mixed<true, false, true, true>(
                E, N, d.M, mixed_src_tile(sb + wid * MixedTile::kBytes, lane),
                mixed_out_tile(mixed_tile(E, (ti.base >> 5) + wid), lane), static_cast<float>(dt1d), dt1d, e, dts, len, ei, eh,
                ev, bad, fo);
        }
        if (live) {
            const PatchArrays PE = d.pa;
            __syncthreads();  // the stage's inputs are consumed
            float* sf = reinterpret_cast<float*>(sb);
            if (e < ne) {
#pragma unroll
                for (int i = 0; i < 24; ++i) sf[i * kPatchElems + tid] = fo[i];
            }
            __syncthreads();
            patch_partials(PE, sf, static_cast<int64_t>(ti.base) / kPatchElems, tid);
        }
        __syncthreads();  // the block is done with stage s
        const int64_t tn = t + 2 * gstride;
        if (tid == 0 && tn < ntiles) {
            const ETileSrc src = *reinterpret_cast<const ETileSrc*>(tail + kBatchNextOff);
            batch_issue<kPatchStageBytes>(T, src, tn + 2 * gstride, ntiles, sb, stage0 + s * SB, bar);
        }
        if (live) batch_tile_sums(T, static_cast<int>(t) * NW + wid, slot, lane, ei, eh, ev, dts, len, bad, &sent[wid]);
    }
    if (timed_out && tid == 0) {
        atomicOr(&T.ctl[T.etile_inst[t]].status, ST_TIMEOUT);
        for (int k = 0; k < 2; ++k) {
            const int itk = it + k;
            if (blockIdx.x + itk * gstride < ntiles) mbar_wait_bounded(bar0 + 8 * (itk & 1), (itk >> 1) & 1);
        }
    }
    element_pass_done(T);
}

// One warp per node tile.  The tile's instance slot and first node are read
// two tiles ahead and its NodeView and NodeParam lines prefetched into L1 one
// tile ahead, so a tile starts on its node rows without waiting on the
// tables.
// NT threads per block (a tuning choice: the warps are independent).
template <int NT, bool PATCH>
__global__ void __launch_bounds__(NT, ENSC_NODE_BATCH_MINB_MIXED * kNodeThreads / NT) k_node_batch_mixed(BatchTables T) {
    constexpr int W = kNodeGroupBatchMixed;
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
                if (PATCH) {
                    node_group_mixed<W, true>(v, dt_i, dt_i_1, amp, n0, kin, wext, bad);
                } else if (v.grouped) {
                    node_group_mixed<W, false>(v, dt_i, dt_i_1, amp, n0, kin, wext, bad);
                } else {
                    const InstanceDesc& d = T.desc[slot];
                    for (int j = 0; j < W && n0 + j < v.nn; ++j)
                        node_body_mixed(d.E, d.N, d.M, dt_i, dt_i_1, amp, n0 + j, kin, wext, bad);
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

void launch_element_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                          int grid, bool init, cudaStream_t st, const PatchArrays& PA) {
    if (PA.pf) {
        if (M.plastic) {
            if (init) k_element_mixed_patch<true, true><<<grid, kPatchElems, kPatchSmem, st>>>(E, N, M, ctl, P, PA);
            else k_element_mixed_patch<true, false><<<grid, kPatchElems, kPatchSmem, st>>>(E, N, M, ctl, P, PA);
        } else {
            if (init) k_element_mixed_patch<false, true><<<grid, kPatchElems, kPatchSmem, st>>>(E, N, M, ctl, P, PA);
            else k_element_mixed_patch<false, false><<<grid, kPatchElems, kPatchSmem, st>>>(E, N, M, ctl, P, PA);
        }
    } else if (M.plastic) {
        if (init) k_element_mixed_init<true><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl);
        else launch_cycle_kernel(k_element_mixed_warp<true>, grid, 32 * kMixedPipeWarps, kMixedPipeSmem, st, E, N, M, ctl, P);
    } else {
        if (init) k_element_mixed_init<false><<<grid, kElemThreads, 0, st>>>(E, N, M, ctl);
        else launch_cycle_kernel(k_element_mixed_warp<false>, grid, 32 * kMixedPipeWarps, kMixedPipeSmem, st, E, N, M, ctl, P);
    }
}

void launch_acceleration_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, const Ctl* ctl,
                               double* a_aos, cudaStream_t st, const PatchArrays& PA) {
    const int64_t g = (N.nn + kNodeThreads - 1) / kNodeThreads;
    k_acceleration_mixed<<<static_cast<int>(g < 65535 ? g : 65535), kNodeThreads, 0, st>>>(PA, E, N, M, ctl, a_aos);
}

void launch_node_mixed(const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl, const Partials& P,
                       int grid, cudaStream_t st, const PatchArrays& PA) {
    if (PA.pf) k_node_mixed<true><<<grid, kNodeThreads, 0, st>>>(E, N, M, ctl, P, PA);
    else k_node_mixed<false><<<grid, kNodeThreads, 0, st>>>(E, N, M, ctl, P, PA);
}

// The pipelined passes need more than the default 48 KB of dynamic shared
// memory; the attribute is set on the current device before any launch or
// capture.
template <typename K>
static int mixed_occupancy(K kernel, int threads, size_t smem) {
    int nb = 0;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem);
    return nb;
}

int occupancy_element_mixed(bool plastic, bool patch) {
    if (patch) {
        // both the init and the cycle pass run
        mixed_occupancy(k_element_mixed_patch<true, true>, kPatchElems, kPatchSmem);
        mixed_occupancy(k_element_mixed_patch<false, true>, kPatchElems, kPatchSmem);
        return plastic ? mixed_occupancy(k_element_mixed_patch<true, false>, kPatchElems, kPatchSmem)
                       : mixed_occupancy(k_element_mixed_patch<false, false>, kPatchElems, kPatchSmem);
    }
    return plastic ? mixed_occupancy(k_element_mixed_warp<true>, 32 * kMixedPipeWarps, kMixedPipeSmem)
                   : mixed_occupancy(k_element_mixed_warp<false>, 32 * kMixedPipeWarps, kMixedPipeSmem);
}

int occupancy_node_mixed() {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_node_mixed<false>, kNodeThreads, 0);
    return nb;
}


void launch_element_batch_mixed(const BatchTables& T, int grid, bool patch, cudaStream_t st) {
    if (patch) launch_cycle_kernel(k_element_batch_patch, grid, kPatchElems, kBatchPatchSmem, st, T);
    else launch_cycle_kernel(k_element_batch_mixed, grid, 32 * kMixedPipeWarps, kBatchMixedSmem, st, T);
}
void launch_node_batch_mixed(const BatchTables& T, int grid, int threads, bool patch, cudaStream_t st) {
    if (patch) {
        if (threads == kNodeThreads / 2) k_node_batch_mixed<kNodeThreads / 2, true><<<grid, threads, 0, st>>>(T);
        else k_node_batch_mixed<kNodeThreads, true><<<grid, kNodeThreads, 0, st>>>(T);
    } else {
        if (threads == kNodeThreads / 2) k_node_batch_mixed<kNodeThreads / 2, false><<<grid, threads, 0, st>>>(T);
        else k_node_batch_mixed<kNodeThreads, false><<<grid, kNodeThreads, 0, st>>>(T);
    }
}
int occupancy_element_batch_mixed(bool patch) {
    // the batch's init passes run the single-instance kernels
    occupancy_element_mixed(true, patch);
    return patch ? mixed_occupancy(k_element_batch_patch, kPatchElems, kBatchPatchSmem)
                 : mixed_occupancy(k_element_batch_mixed, 32 * kMixedPipeWarps, kBatchMixedSmem);
}

RunPlan plan_run_mixed(int64_t ne, int64_t nn, bool plastic, int sms) {
    return plastic ? plan_run(k_run_mixed<true, true, 1>, k_run_mixed<true, true, 2>, k_run_mixed<true, false, 1>,
                              k_run_mixed<true, false, 2>, ne, nn, sms, kRunWarpsMixed, RunMixed<true>::kTileBytes)
                   : plan_run(k_run_mixed<false, true, 1>, k_run_mixed<false, true, 2>, k_run_mixed<false, false, 1>,
                              k_run_mixed<false, false, 2>, ne, nn, sms, kRunWarpsMixed, RunMixed<false>::kTileBytes);
}
cudaError_t launch_run_mixed(const RunPlan& p, const ElemArrays& E, const NodeArrays& N, const Material& M, Ctl* ctl,
                             const Partials& P, RunSync* sync, const RunArgs& a, cudaStream_t st) {
    using K = void (*)(ElemArrays, NodeArrays, Material, Ctl*, Partials, RunSync*, RunArgs);
    static const K kernels[8] = {k_run_mixed<false, false, 1>, k_run_mixed<false, false, 2>,
                                 k_run_mixed<false, true, 1>,  k_run_mixed<false, true, 2>,
                                 k_run_mixed<true, false, 1>,  k_run_mixed<true, false, 2>,
                                 k_run_mixed<true, true, 1>,   k_run_mixed<true, true, 2>};
    return launch_run(kernels[(M.plastic ? 4 : 0) + (p.cluster ? 2 : 0) + p.node_width - 1], p, st, E, N, M, ctl, P,
                      sync, a);
}

int batch_element_tile(bool patch) { return patch ? kPatchElems : 32; }
int batch_node_tile(bool mixed_precision) { return 32 * (mixed_precision ? kNodeGroupBatchMixed : kNodeGroupFp64); }
int occupancy_node_batch_mixed(int threads) {
    int nb = 0;
    if (threads == kNodeThreads / 2)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_node_batch_mixed<kNodeThreads / 2, false>, threads, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_node_batch_mixed<kNodeThreads, false>, kNodeThreads, 0);
    return nb;
}

}  // namespace ensc
