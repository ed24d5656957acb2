// joints.cuh — device helpers for joint rows (ball-socket, hinge, distance,
// weld, slider, sliding hinge, cone and twist limits, motors, pistons) and the holonomic block
// solve, shared by the row-building kernels (joints.cu) and
// the joint-island PGS kernel (solver.cu).
#pragma once
#include "devmath.cuh"
#include "layout.h"

namespace cpgpu {

constexpr float kJZero = 0.00000001f;   // NVec::isZero cutoff (Math/src/NVec.h:4)

// Δv slots of one island: kDvF4 float4 per island body, 12 floats v xyz,
// w xyz, pv xyz, pw xyz; `which` 0 = (v, w), 1 = (pv, pw)
__device__ __forceinline__ void jload(const float4* dv, int slot, int which, float* out) {
    if (slot < 0) { for (int k = 0; k < 6; k++) out[k] = 0.f; return; }
    const float* f = reinterpret_cast<const float*>(dv + kDvF4 * slot) + 6 * which;
    for (int k = 0; k < 6; k++) out[k] = f[k];
}
// J_a v_a + J_b v_b
__device__ __forceinline__ void jvalue(const JointRow& R, const float* va, const float* vb, float* out) {
    for (int i = 0; i < R.n; i++) {
        float x = 0.f, y = 0.f;
        for (int k = 0; k < 6; k++) x += va[k] * R.ja[6 * i + k];
        for (int k = 0; k < 6; k++) y += vb[k] * R.jb[6 * i + k];
        out[i] = x + y;
    }
}

// ---- one joint row by a warp ----------------------------------------------------
// A row's work is spread over lanes so that a row-step is a few short chains
// instead of a few hundred instructions on one lane: lane i < 6 has dof i (its
// two Jacobian rows and its row of the effective mass inverse), lane c < 12
// component c of M^-1 J^T and of the two bodies' Δv (a's six, then b's); lanes
// meet by shuffles.  Every sum runs in the order of the one-thread form with
// FMAs from zero, so the results are the same bits; dofs beyond the row's are
// zeros.  Loaded one row ahead of its use.  (The passes over the rows are
// joint_pass in solver.cu; here is what the block solve shares with them.)
struct JointLane {
    float it[6];   // component lane
    int n, sa, sb;
};
__device__ __forceinline__ void jl_row6(const float* p, float* o) {   // 8-byte aligned
    const float2* q = reinterpret_cast<const float2*>(p);
    const float2 x = q[0], y = q[1], z = q[2];
    o[0] = x.x; o[1] = x.y; o[2] = y.x; o[3] = y.y; o[4] = z.x; o[5] = z.y;
}
__device__ __forceinline__ void jl_load(const JointRow& R, int lane, JointLane& L) {
    L.n = R.n; L.sa = R.sa; L.sb = R.sb;
    jl_row6(R.ita + kJMax * min(lane, 11), L.it);   // body b's follow body a's
}
// component lane: sum of imp_i M^-1 J^T added to its component of Δv, where
// lane i holds imp_i (finite beyond the row's dofs)
__device__ __forceinline__ void jl_apply(const JointLane& L, float imp, float4* dv, int which, int lane) {
    const int slot = lane < 6 ? L.sa : L.sb;
    float x = 0.f;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        x = __fmaf_rn(__shfl_sync(0xffffffffu, imp, i), L.it[i], x);
    }
    if (lane < 12 && slot >= 0) {
        float* f = reinterpret_cast<float*>(dv + kDvF4 * slot) + 6 * which + (lane < 6 ? lane : lane - 6);
        *f = __fadd_rn(*f, x);
    }
    __syncwarp();
}

// ---- holonomic systems (HolonomicBlockSolver.cpp) ------------------------------
__device__ __forceinline__ int holo_loc(const int* table, int n, int row, int col) {
    return table[row - col + ((2 * n + 1) * col - col * col) / 2];
}

// The tables of one system as the solve reads them: in shared memory when the
// system is small enough (each column's solve is a chain of dependent loads),
// else where the host put them.
struct HoloView {
    int n;
    const int *cons, *vpos, *ls, *lrow, *lloc;   // ls: column col's blocks below the diagonal, [ls[col], ls[col + 1]) - ls0
    const int* dim;                              // dofs per constraint
    int ls0;
};
__device__ __forceinline__ double jfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float jfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// multInverseWithVector (HolonomicBlockSolver.cpp:251-317): v <- L^-T D^-1 L^-1 v
// by one warp, a lane per entry of the blocks of a column (each entry summed in
// the order of the one-thread form); the next column's first blocks are loaded
// while this one is solved.
template <class T>
__device__ __forceinline__ void holo_solve(const HoloView& h, const int* table, const T* B, T* v, int lane) {
    const int n = h.n;
    const int r8 = lane >> 3, i8 = lane & 7;   // four blocks at a time, eight lanes each
    T b[kJMax], nb[kJMax];
    int row = 0, nrow = 0;
    bool act = false, nact = false;
    auto lower = [&](int col, int q, T* o, int* r) {   // block q's row i8
        bool a = q < h.ls[col + 1] - h.ls0;
        *r = a ? h.lrow[q] : 0;
        a = a && i8 < h.dim[*r];
        const int bw = h.dim[col], l = a ? h.lloc[q] : 0;
#pragma unroll
        for (int k = 0; k < kJMax; k++) o[k] = a && k < bw ? B[l + i8 * bw + k] : (T)0;
        return a;
    };
    if (n > 1) act = lower(0, h.ls[0] - h.ls0 + r8, b, &row);
    for (int col = 0; col + 1 < n; col++) {
        const int bw = h.dim[col];
        const T* vc = v + h.vpos[col];
        if (col + 2 < n) nact = lower(col + 1, h.ls[col + 1] - h.ls0 + r8, nb, &nrow);
        T x = 0;
#pragma unroll
        for (int k = 0; k < kJMax; k++) x = k < bw ? jfma(b[k], vc[k], x) : x;
        if (act) v[h.vpos[row] + i8] -= x;
        for (int q0 = h.ls[col] - h.ls0 + 4; q0 < h.ls[col + 1] - h.ls0; q0 += 4) {   // more than four blocks
            T c[kJMax];
            int r;
            if (lower(col, q0 + r8, c, &r)) {
                T y = 0;
                for (int k = 0; k < bw; k++) y = jfma(c[k], vc[k], y);
                v[h.vpos[r] + i8] -= y;
            }
        }
        __syncwarp();
        act = nact;
        row = nrow;
#pragma unroll
        for (int k = 0; k < kJMax; k++) b[k] = nb[k];
    }
    for (int col = r8; col < n; col += 4) {
        const int w = h.dim[col], l = holo_loc(table, n, col, col);
        T x = 0;
        if (i8 < w)
            for (int k = 0; k < w; k++) x = jfma(B[l + i8 * w + k], v[h.vpos[col] + k], x);
        __syncwarp(0xffu << (lane & 24));   // the eight lanes of the block
        if (i8 < w) v[h.vpos[col] + i8] = x;
    }
    __syncwarp();
    auto upper = [&](int col, int q, T* o, int* r) {   // block q's column `lane`
        const bool a = q < h.ls[col + 1] - h.ls0;
        *r = a ? h.lrow[q] : 0;
        const int bw = h.dim[col], bh = a ? h.dim[*r] : 0, l = a ? h.lloc[q] : 0;
#pragma unroll
        for (int j = 0; j < kJMax; j++) o[j] = lane < bw && j < bh ? B[l + lane + bw * j] : (T)0;
        return bh;
    };
    int bh = 0, nbh = 0;
    if (n > 1) bh = upper(n - 2, h.ls[n - 2] - h.ls0, b, &row);
    for (int col = n - 2; col >= 0; col--) {
        const int bw = h.dim[col];
        if (col > 0) nbh = upper(col - 1, h.ls[col - 1] - h.ls0, nb, &nrow);
        if (lane < bw) {
            T e = 0;
            T dp = 0;
            const T* vr = v + h.vpos[row];
#pragma unroll
            for (int j = 0; j < kJMax; j++) dp = j < bh ? jfma(vr[j], b[j], dp) : dp;
            if (h.ls[col] < h.ls[col + 1]) e += dp;
            for (int q = h.ls[col] - h.ls0 + 1; q < h.ls[col + 1] - h.ls0; q++) {
                const int r = h.lrow[q], l = h.lloc[q];
                const int rh = h.dim[r];
                T y = 0;
                for (int j = 0; j < rh; j++) y = jfma(v[h.vpos[r] + j], B[l + lane + bw * j], y);
                e += y;
            }
            v[h.vpos[col] + lane] -= e;
        }
        __syncwarp();
        bh = nbh;
        row = nrow;
#pragma unroll
        for (int j = 0; j < kJMax; j++) b[j] = nb[j];
    }
}

}  // namespace cpgpu
