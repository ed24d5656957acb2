// solver.cu — per-substep row rebuild, projected Gauss-Seidel and integration.
//
// Rows (Contact::updateSolverConstraints, PersistentConstraint.cpp:201-215;
// ContactConstraint / FrictionConstraint constructors, ConstraintSolver.cpp:
// 240-343): one thread per live contact rebuilds its normal row and 2-dof
// friction row from the current poses and writes them, with the warm-start
// impulses (the friction impulse re-projected onto the new tangent basis), to
// the contact's slot in island order.  The same pass advances the contact's
// lifetime (PhysicsEngine.cpp:1378-1399) and marks expired contacts.
//
// PGS (PGS_solve, ConstraintSolver.cpp:80-213): each island's rows one after the
// other in the reference's order: targets from the bodies' velocities, warm
// start, n_vel velocity sweeps of block Gauss-Seidel with the projection on the
// accumulated impulse, n_pos pseudo-velocity sweeps of the normal rows, then the
// velocity deltas are applied to the island's bodies.  A large or middling island
// takes two lanes of a warp (a body of the contact each), one with joints a
// warp, a small one a thread.  A serial chain per island is the latency-optimal
// form of Gauss-Seidel (each row depends on the previous one); throughput comes
// from running thousands of islands at once.
//
// Integration (PhysicsEngine.cpp:390-419, RigidBody.cpp:207-279): one thread
// per body.
#include <algorithm>

#include "kernels.cuh"
#include "devmath.cuh"
#include "shapes.cuh"
#include "joints.cuh"

namespace cpgpu {

namespace {

constexpr float kZero = 0.00000001f;  // NVec::isZero cutoff (Math/src/NVec.h:4)

__device__ __forceinline__ f3 qrotate(float4 q, f3 v) {  // Quaternion::applyRotation
    float r = q.x, i = q.y, j = q.z, k = q.w;
    return mk(v.x * (r * r + i * i - j * j - k * k) + v.y * (2 * i * j - 2 * r * k) + v.z * (2 * i * k + 2 * r * j),
              v.x * (2 * i * j + 2 * r * k) + v.y * (r * r - i * i + j * j - k * k) + v.z * (2 * j * k - 2 * r * i),
              v.x * (2 * i * k - 2 * r * j) + v.y * (2 * j * k + 2 * r * i) + v.z * (r * r - i * i - j * j + k * k));
}

// J angular part n^T [r]x (ConstraintSolver.cpp:247-252)
__device__ __forceinline__ f3 nskew(f3 n, f3 r) {
    return mk(n.y * r.z - n.z * r.y, n.z * r.x - n.x * r.z, n.x * r.y - n.y * r.x);
}

__device__ __forceinline__ void it_of(float im, const M33& I, const float* j, float* out) {
    out[0] = im * j[0]; out[1] = im * j[1]; out[2] = im * j[2];
    f3 a = mul(I, mk(j[3], j[4], j[5]));
    out[3] = a.x; out[4] = a.y; out[5] = a.z;
}

__device__ __forceinline__ float dot6(const float* a, const float* b) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 6; k++) s += a[k] * b[k];
    return s;
}

__device__ __forceinline__ void body_vel(const Dev& d, int g, float* out) {
    if (d.movement[g] == 1) { for (int k = 0; k < 6; k++) out[k] = 0.f; return; }
    float4 v = d.vel[g], w = d.angv[g];
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = w.x; out[4] = w.y; out[5] = w.z;
}

__global__ void k_rows(Dev d, int first, int last) {
    const int nc = *d.n_contacts_new;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        int st = d.c_new.state[c];
        const bool live = cs_live(st);
        const int r = live ? d.row_of_contact[c] : -1;
        if (live && r >= 0) {
            const uint64_t key = d.e_new.key[d.c_new.edge[c]];
            const int a = (int)(key >> 32), b = (int)(key & 0xffffffffu);
            const WorldParams& P = d.wparams[d.world[a]];
            const float dt = P.dt_sub;
            const float4 qa = d.rot[a], qb = d.rot[b];
            const f3 ca = mk(d.pos[a]), cb = mk(d.pos[b]);
            const float ima = d.pos[a].w, imb = d.pos[b].w;
            const M33 Ia = load9(d.iinv + 9 * a), Ib = load9(d.iinv + 9 * b);
            const float4 p1 = d.c_new.p1[c], p2 = d.c_new.p2[c], nl = d.c_new.n[c], imp = d.c_new.imp[c];
            const f3 pa = qrotate(qa, mk(p1)) + ca;
            const f3 pb = qrotate(qb, mk(p2)) + cb;
            const f3 n = qrotate(qa, mk(nl));
            const float depth = dot(pb - pa, n) + p1.w;
            const float wn = P.warm_disabled ? 0.f : imp.x;
            const float wf0 = P.warm_disabled ? 0.f : imp.y, wf1 = P.warm_disabled ? 0.f : imp.z;
            const float pcc = fminf(P.hardness * dt, 1.0f / dt);
            const f3 rA = pa - ca, rB = pa - cb;
            // the row is assembled in registers and written with 16-byte stores
            // (a thread per contact writing 384 scattered bytes field by field
            // would issue 96 partial-sector stores)
            RowBlock R;
            R.sa = (d.movement[a] == 0) ? d.visited[a] : -1;
            R.sb = (d.movement[b] == 0) ? d.visited[b] : -1;
            R.contact = c;
            R.ga = a; R.gb = b;
            R.bounce = p2.w;
            R.cutoff = P.cutoff_vel;
            R.fcoeff = nl.w;
            R.stat = 0;
            // normal row
            float ja[6], jb[6], ia[6], ib[6];
            f3 t = nskew(n, rA), t2 = nskew(-n, rB);
            ja[0] = -n.x; ja[1] = -n.y; ja[2] = -n.z; ja[3] = t.x; ja[4] = t.y; ja[5] = t.z;
            jb[0] = n.x; jb[1] = n.y; jb[2] = n.z; jb[3] = t2.x; jb[4] = t2.y; jb[5] = t2.z;
            it_of(ima, Ia, ja, ia);
            it_of(imb, Ib, jb, ib);
            float itv = dot6(ja, ia) + dot6(jb, ib);
            for (int k = 0; k < 6; k++) { R.a.nj[k] = ja[k]; R.b.nj[k] = jb[k]; R.a.nit[k] = ia[k]; R.b.nit[k] = ib[k]; }
            R.nminv = 1.0f / (itv * (1.0f + P.cfm));
            R.nptarget = fmaxf(0.0f, depth - 0.05f) * pcc;
            // friction rows in the tangent basis of n, warm impulse re-projected
            f3 u, w;
            basis(n, &u, &w);
            const f3 su = mk(d.c_new.fu[c]), sw = mk(d.c_new.fw[c]);
            R.imp = make_float4(wn, 0.f, dot(u, su) * wf0 + dot(u, sw) * wf1, dot(w, su) * wf0 + dot(w, sw) * wf1);
            float fja[12], fjb[12], fia[12], fib[12];
            f3 ta = nskew(-u, rA), tb = nskew(u, rB), wa = nskew(-w, rA), wb = nskew(w, rB);
            fja[0] = u.x; fja[1] = u.y; fja[2] = u.z; fja[3] = ta.x; fja[4] = ta.y; fja[5] = ta.z;
            fja[6] = w.x; fja[7] = w.y; fja[8] = w.z; fja[9] = wa.x; fja[10] = wa.y; fja[11] = wa.z;
            fjb[0] = -u.x; fjb[1] = -u.y; fjb[2] = -u.z; fjb[3] = tb.x; fjb[4] = tb.y; fjb[5] = tb.z;
            fjb[6] = -w.x; fjb[7] = -w.y; fjb[8] = -w.z; fjb[9] = wb.x; fjb[10] = wb.y; fjb[11] = wb.z;
            float tmp[6];
            for (int row = 0; row < 2; row++) {
                it_of(ima, Ia, fja + 6 * row, tmp);
                for (int k = 0; k < 6; k++) fia[2 * k + row] = tmp[k];
                it_of(imb, Ib, fjb + 6 * row, tmp);
                for (int k = 0; k < 6; k++) fib[2 * k + row] = tmp[k];
            }
            float fv[4];
            for (int i = 0; i < 2; i++)
                for (int j = 0; j < 2; j++) {
                    float sa = 0.f, sb = 0.f;
                    for (int k = 0; k < 6; k++) { sa += fja[6 * i + k] * fia[2 * k + j]; sb += fjb[6 * i + k] * fib[2 * k + j]; }
                    fv[2 * i + j] = sa + sb;
                }
            fv[0] *= (1.0f + P.cfm);
            fv[3] *= (1.0f + P.cfm);
            float di = 1.0f / (fv[0] * fv[3] - fv[1] * fv[2]);
            const float m00 = fv[3] * di, m01 = -fv[1] * di, m10 = -fv[2] * di, m11 = fv[0] * di;
            R.fmc[0] = m00; R.fmc[1] = m10; R.fmc[2] = m01; R.fmc[3] = m11;
            // the friction values' change per unit normal impulse (J_f M^-1 J_n^T),
            // mapped through Fm^-1 to the friction impulses' change
            const float kf0 = dot6(fja, ia) + dot6(fjb, ib);
            const float kf1 = dot6(fja + 6, ia) + dot6(fjb + 6, ib);
            R.kd0 = m00 * kf0 + m01 * kf1;
            R.kd1 = m10 * kf0 + m11 * kf1;
            for (int k = 0; k < 6; k++) {
                R.a.fj0[k] = fja[k]; R.b.fj0[k] = fjb[k]; R.a.fj1[k] = fja[6 + k]; R.b.fj1[k] = fjb[6 + k];
                R.a.fit0[k] = fia[2 * k]; R.b.fit0[k] = fib[2 * k]; R.a.fit1[k] = fia[2 * k + 1]; R.b.fit1[k] = fib[2 * k + 1];
            }
            // velocity targets from the bodies' velocities at the start of the
            // solve (ContactConstraint::findTargetConstraintValue,
            // ConstraintSolver.cpp:264-268; DegreedConstraint default, ConstraintSolver.h:78)
            {
                float va[6], vb[6];
                body_vel(d, a, va);
                body_vel(d, b, vb);
                float cur = dot6(ja, va) + dot6(jb, vb);
                R.tgt_n = (cur < -P.cutoff_vel) ? -(1.0f + p2.w) * cur : -cur;
                R.tgt_f0 = -(dot6(fja, va) + dot6(fjb, vb));
                R.tgt_f1 = -(dot6(fja + 6, va) + dot6(fjb + 6, vb));
            }
            {
                float4* dst = reinterpret_cast<float4*>(d.rows + r);
                const float4* src = reinterpret_cast<const float4*>(&R);
#pragma unroll
                for (int k = 0; k < (int)(sizeof(RowBlock) / 16); k++) dst[k] = src[k];
            }
            d.c_new.fu[c] = make_float4(u.x, u.y, u.z, 0.f);
            d.c_new.fw[c] = make_float4(w.x, w.y, w.z, 0.f);
        }
        // lifetime (PhysicsEngine.cpp:1378-1399, expiry :1434-1446)
        int life = cs_life(st);
        bool lv = live;
        if (last) { life = life > -127 ? life - 1 : life; lv = false; }   // the 8-bit store saturates
        bool dead = cs_dead(st) || (first && life < 0);
        if (dead && !cs_dead(st) && d.has_sleep) {
            // Contact::isExpired (PersistentConstraint.h:74): a contact of a
            // sleeping body does not expire
            const uint64_t key = d.e_new.key[d.c_new.edge[c]];
            if (d.asleep[(int)(key >> 32)] || d.asleep[(int)(key & 0xffffffffu)]) dead = false;
        }
        // a rebuilt FrictionConstraint starts with static_ready = false
        d.c_new.state[c] = cs_make(life, lv, live ? false : cs_static(st), dead);
    }
}

// ---- packed FP32 pairs: a row's 6-vectors and a body's Δv are handled as
// the three component pairs (x, y), (z, ax), (ay, az), two lanes of one
// fma.rn.f32x2 each (half the instructions of scalar FP32 on the chain).
// Every operation of the rows is written with an explicit round-to-nearest
// intrinsic: the row functions are inlined into several kernels (warp per
// island, thread per island, joint islands), and left to the compiler, a
// sum of two products could be contracted into a different FMA in each;
// spelled out, every kernel computes the same bits, so the island-size
// threshold between the kernels never changes a result.
struct P3 { float2 a, b, c; };
__device__ __forceinline__ P3 p3(const float* f) {
    return P3{make_float2(f[0], f[1]), make_float2(f[2], f[3]), make_float2(f[4], f[5])};
}
__device__ __forceinline__ float2 bc2(float x) { return make_float2(x, x); }
// x - y, rounded once (y times -1 is exact)
__device__ __forceinline__ float2 psub(float2 x, float2 y) { return __ffma2_rn(y, make_float2(-1.f, -1.f), x); }
// J_a v_a + J_b v_b
__device__ __forceinline__ float pdot(const P3& ja, const P3& va, const P3& jb, const P3& vb) {
    float2 s = __fmul2_rn(ja.a, va.a);
    s = __ffma2_rn(ja.b, va.b, s);
    s = __ffma2_rn(ja.c, va.c, s);
    float2 t = __fmul2_rn(jb.a, vb.a);
    t = __ffma2_rn(jb.b, vb.b, t);
    t = __ffma2_rn(jb.c, vb.c, t);
    const float2 u = __fadd2_rn(s, t);
    return __fadd_rn(u.x, u.y);
}
// v += x * s
__device__ __forceinline__ void paxpy(P3& v, const P3& x, float2 s) {
    v.a = __ffma2_rn(x.a, s, v.a);
    v.b = __ffma2_rn(x.b, s, v.b);
    v.c = __ffma2_rn(x.c, s, v.c);
}

// Δv of island body `slot`: which 0 = (v, w), 1 = (pv, pw); slot < 0 is a
// body of infinite mass (always zero)
__device__ __forceinline__ P3 dv_get_z(const float4* dv, int slot, int which) {   // dv has an entry at -1
    const float4* s = dv + kDvF4 * slot;
    if (which == 0) {
        const float4 A = s[0];
        const float2 B = reinterpret_cast<const float2*>(s + 1)[0];
        return P3{make_float2(A.x, A.y), make_float2(A.z, A.w), B};
    }
    const float2 A = reinterpret_cast<const float2*>(s + 1)[1];
    const float4 C = s[2];
    return P3{A, make_float2(C.x, C.y), make_float2(C.z, C.w)};
}
__device__ __forceinline__ P3 dv_get(const float4* dv, int slot, int which) {
    if (slot < 0) return P3{make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    return dv_get_z(dv, slot, which);
}
__device__ __forceinline__ void dv_put_z(float4* dv, int slot, int which, const P3& v) {
    float4* s = dv + kDvF4 * slot;
    if (which == 0) {
        s[0] = make_float4(v.a.x, v.a.y, v.b.x, v.b.y);
        reinterpret_cast<float2*>(s + 1)[0] = v.c;
    } else {
        reinterpret_cast<float2*>(s + 1)[1] = v.a;
        s[2] = make_float4(v.b.x, v.b.y, v.c.x, v.c.y);
    }
}

__device__ __forceinline__ void dv_put(float4* dv, int slot, int which, const P3& v) {
    if (slot >= 0) dv_put_z(dv, slot, which, v);
}

// ---- one row of each PGS pass (PGS_solve, ConstraintSolver.cpp:120-161) ----------
// warm start: apply the stored impulses when they are non-zero
// (DegreedConstraint::constraintWarmStarted / applyWarmStartVelocityChange)
__device__ __forceinline__ void row_warm(const RowBlock& R, const float4 imp, float4* dv) {
    const bool wn = fabsf(imp.x) > kZero, wf = fabsf(imp.z) > kZero || fabsf(imp.w) > kZero;
    if (!wn && !wf) return;
    P3 va = dv_get(dv, R.sa, 0), vb = dv_get(dv, R.sb, 0);
    if (wn) {
        paxpy(va, p3(R.a.nit), bc2(imp.x));
        paxpy(vb, p3(R.b.nit), bc2(imp.x));
    }
    if (wf) {
        paxpy(va, p3(R.a.fit0), bc2(imp.z));
        paxpy(va, p3(R.a.fit1), bc2(imp.w));
        paxpy(vb, p3(R.b.fit0), bc2(imp.z));
        paxpy(vb, p3(R.b.fit1), bc2(imp.w));
    }
    dv_put(dv, R.sa, 0, va);
    dv_put(dv, R.sb, 0, vb);
}

// velocity pass: normal row clamped at zero, then the friction rows projected on
// the friction disc of the current normal impulse (PGSConstraintStep,
// ConstraintSolver.cpp:12-40; projections :270-272, :331-343).  The friction
// rows see the velocities after the normal change; their new impulses are
// evaluated as (impulses + Fm^-1 (targets - values of the incoming
// velocities)) minus the normal change times the row's constants
// kd = Fm^-1 J_f M^-1 J_n^T (the same quantity, associated differently), so
// that everything but one FMA per friction row runs alongside the normal row
// instead of after it; the normal row's velocity change is applied while the
// friction rows are evaluated.  The disc projection compares squared
// magnitudes and scales by rsqrt.  `va`, `vb` are the two bodies' Δv.
__device__ __forceinline__ void row_vel_r(const RowBlock& R, float4& imp, int& stat, P3& va, P3& vb) {
    const float cur = pdot(p3(R.a.nj), va, p3(R.b.nj), vb);
    const float b0 = pdot(p3(R.a.fj0), va, p3(R.b.fj0), vb), b1 = pdot(p3(R.a.fj1), va, p3(R.b.fj1), vb);
    // friction impulses for the incoming velocities: imp.zw + Fm^-1 (tgt_f - b)
    const float2 g = psub(make_float2(R.tgt_f0, R.tgt_f1), make_float2(b0, b1));
    const float2 A = __fadd2_rn(make_float2(imp.z, imp.w),
                                __ffma2_rn(make_float2(R.fmc[2], R.fmc[3]), bc2(g.y),
                                           __fmul2_rn(make_float2(R.fmc[0], R.fmc[1]), bc2(g.x))));
    const float nw = __fmaf_rn(R.nminv, __fsub_rn(R.tgt_n, cur), imp.x);
    float diff = __fsub_rn(fmaxf(nw, 0.0f), imp.x);
    if (!(fabsf(diff) > kZero)) diff = 0.f;
    const float ix = __fadd_rn(imp.x, diff);
    const float2 sd = bc2(diff);
    paxpy(va, p3(R.a.nit), sd);
    paxpy(vb, p3(R.b.nit), sd);
    float2 nf = __ffma2_rn(bc2(-diff), make_float2(R.kd0, R.kd1), A);
    const float mx = __fmul_rn(R.fcoeff, ix);
    const float s2 = __fmaf_rn(nf.x, nf.x, __fmul_rn(nf.y, nf.y));
    if (s2 > __fmul_rn(mx, mx)) { nf = __fmul2_rn(nf, bc2(__fmul_rn(mx, rsqrtf(s2)))); stat = 0; }
    else stat = 1;
    float2 e = psub(nf, make_float2(imp.z, imp.w));
    if (!(fabsf(e.x) > kZero || fabsf(e.y) > kZero)) e = make_float2(0.f, 0.f);
    const float2 s0 = bc2(e.x), s1 = bc2(e.y);
    paxpy(va, p3(R.a.fit0), s0);
    paxpy(vb, p3(R.b.fit0), s0);
    paxpy(va, p3(R.a.fit1), s1);
    paxpy(vb, p3(R.b.fit1), s1);
    imp.x = ix;
    imp.z = __fadd_rn(imp.z, e.x);
    imp.w = __fadd_rn(imp.w, e.y);
}
// the same on the island's Δv array (written back unconditionally: a zero
// change writes the same values)
__device__ __forceinline__ void row_vel(const RowBlock& R, float4& imp, int& stat, float4* dv) {
    P3 va = dv_get(dv, R.sa, 0), vb = dv_get(dv, R.sb, 0);
    row_vel_r(R, imp, stat, va, vb);
    dv_put(dv, R.sa, 0, va);
    dv_put(dv, R.sb, 0, vb);
}

// pseudo-velocity (position correction) pass of the normal row
__device__ __forceinline__ void row_pos(const RowBlock& R, float4& imp, float4* dv) {
    P3 va = dv_get(dv, R.sa, 1), vb = dv_get(dv, R.sb, 1);
    const float cur = pdot(p3(R.a.nj), va, p3(R.b.nj), vb);
    const float nw = __fmaf_rn(R.nminv, __fsub_rn(R.nptarget, cur), imp.y);
    const float diff = __fsub_rn(fmaxf(nw, 0.0f), imp.y);
    if (fabsf(diff) > kZero) {
        paxpy(va, p3(R.a.nit), bc2(diff));
        paxpy(vb, p3(R.b.nit), bc2(diff));
        imp.y = __fadd_rn(imp.y, diff);
        dv_put(dv, R.sa, 1, va);
        dv_put(dv, R.sb, 1, vb);
    }
}

// island epilogue: impulses to the contacts (warm start of the next rebuild)
// and velocity deltas to the bodies (PhysicsEngine::applyVelocityChange,
// PhysicsEngine.cpp:1113-1136); `t`/`nt` stride over the island
__device__ void island_finish(const Dev& d, int rs, int rc, int bs, int bc, const float4* dv, int t, int nt) {
    for (int r = rs + t; r < rs + rc; r += nt) {
        const RowBlock& R = d.rows[r];
        if (R.contact < 0) continue;   // joint row (k_pgs_joint writes those back)
        float4 imp = R.imp;
        d.c_new.imp[R.contact] = make_float4(imp.x, imp.z, imp.w, 0.f);
        int cst = d.c_new.state[R.contact];
        d.c_new.state[R.contact] = R.stat ? (cst | (1 << 9)) : (cst & ~(1 << 9));
    }
    bool wake = false;
    for (int k = t; k < bc; k += nt) {
        int g = d.isl_bodies[bs + k];
        if (d.movement[g] != 0) continue;
        const float4 A = dv[kDvF4 * k], B = dv[kDvF4 * k + 1], C = dv[kDvF4 * k + 2];
        float4 v = d.vel[g], w = d.angv[g], pv = d.pvel[g], pw = d.pangv[g];
        v = make_float4(v.x + A.x, v.y + A.y, v.z + A.z, 0.f);
        w = make_float4(w.x + A.w, w.y + B.x, w.z + B.y, 0.f);
        d.vel[g] = v;
        d.angv[g] = w;
        d.pvel[g] = make_float4(pv.x + B.z, pv.y + B.w, pv.z + C.x, 0.f);
        d.pangv[g] = make_float4(pw.x + C.y, pw.y + C.z, pw.z + C.w, 0.f);
        if (d.has_sleep && d.asleep[g]) {
            const float wv = d.wparams[d.world[g]].wake_vel;
            wake = wake || mag(mk(v)) > wv || mag(mk(w)) > wv;
        }
    }
    if (!d.has_sleep) return;
    // sleeping bodies of a solved island (PhysicsEngine::applyVelocityChange,
    // PhysicsEngine.cpp:1113-1136): one pushed faster than a quarter of the
    // sleep velocity wakes the island (the island is the component
    // wakeupIsland walks); otherwise they keep zero velocity.  The reference
    // visits the bodies in an unordered_map's order, and a body zeroed before
    // the waking one stays at rest there; here a wake takes precedence.
    if (nt == 32) wake = __any_sync(0xffffffffu, wake);
    for (int k = t; k < bc; k += nt) {
        const int g = d.isl_bodies[bs + k];
        if (d.movement[g] != 0 || !d.asleep[g]) continue;
        if (wake) {
            d.asleep[g] = 0;
            d.ready_cnt[g] = 0;
            d.non_sleepy[g] = 0;
            d.hist_n[g] = 0;
            d.hist_head[g] = 0;
        } else {
            d.vel[g] = make_float4(0.f, 0.f, 0.f, 0.f);
            d.angv[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

// ---- scheduling: islands with at least d.big_rows rows get a warp each,
// largest first; middling ones a warp with all their rows in shared memory, the
// smaller ones a thread each (the three paths give identical results, so the
// thresholds are pure schedule choices)

// sched[kLongIslands]: islands of at least 2^kLongBucket rows
constexpr int kLongIslands = 4, kLongBucket = 9;
// islands of kMidRows to kMidMax rows below the big ones: sched[kMidIslands];
// from kMidRowsFew rows in a batch of up to kMidFew islands
constexpr int kMidIslands = 5, kMidRows = 16, kMidMax = 48, kMidRowsFew = 4, kMidFew = 8192;
// a big_rows that no island reaches (the caller wants no island on a warp): from
// here up the middling class is off too
constexpr int kNoWarps = 1 << 20;
__device__ __forceinline__ int size_bucket(int rows) { return 31 - __clz(rows); }

__global__ void k_sched_count(Dev d) {
    const int ni = *d.n_islands;
    const int mid = d.big_rows >= kNoWarps ? kMidMax + 1 : ni <= kMidFew ? kMidRowsFew : kMidRows;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ni; i += gridDim.x * blockDim.x) {
        if (d.n_joint_edges > 0 && d.g_isl_flags[i]) { d.joint_list[atomicAdd(&d.sched[3], 1)] = i; continue; }
        int rc = d.g_isl_row_count[i];
        if (rc >= d.big_rows) atomicAdd(&d.sched[32 + size_bucket(rc)], 1);
        else if (rc >= mid && rc <= kMidMax && d.g_isl_body_count[i] <= kMidMax + 1) d.big_list[d.n_bodies - 1 - atomicAdd(&d.sched[kMidIslands], 1)] = i;   // from the list's end
        else d.small_list[atomicAdd(&d.sched[1], 1)] = i;
    }
}

__global__ void k_sched_place(Dev d) {
    const int ni = *d.n_islands;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ni; i += gridDim.x * blockDim.x) {
        if (d.n_joint_edges > 0 && d.g_isl_flags[i]) continue;
        int rc = d.g_isl_row_count[i];
        if (rc < d.big_rows) continue;
        int b = size_bucket(rc), off = 0;
        for (int k = 31; k > b; k--) off += d.sched[32 + k];   // larger buckets first
        d.big_list[off + atomicAdd(&d.sched[64 + b], 1)] = i;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        int n = 0, lng = 0;
        for (int k = 0; k < 32; k++) {
            n += d.sched[32 + k];
            if (k >= kLongBucket) lng += d.sched[32 + k];
        }
        d.sched[0] = n;
        d.sched[kLongIslands] = lng;
    }
}

// small islands: one thread walks the island's rows in global memory.  Islands
// are dealt to the warps in turn, so that a warp holds a few lanes' scattered
// rows instead of 32 (6,300 islands of a world of 20,000 bodies: 1,203 -> 466
// us); but to consecutive threads of half the blocks when there are more of
// them than that (150,000 islands: 652 us, dealt out 1,217), or when a chain
// of 512 rows or more bounds the step anyway: the fewer warps then slow that
// chain less (96 served worlds 75 ms, dealt out 80).
__global__ void k_pgs_small(Dev d) {
    const int n = d.sched[1];
    const int nt = gridDim.x * blockDim.x, nw = nt >> 5;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, warp = tid >> 5;
    const bool dense = 2 * n > nt || d.sched[kLongIslands] > 0;
    if (dense && 2 * blockIdx.x >= gridDim.x) return;
    const int step = dense ? nt / 2 : nt;
    for (int q = dense ? tid : warp + nw * (threadIdx.x & 31); q < n; q += step) {
        const int i = d.small_list[q];
        const int rs = d.g_isl_row_start[i], rc = d.g_isl_row_count[i];
        const int bs = d.g_isl_body_start[i], bc = d.g_isl_body_count[i];
        const WorldParams& P = d.wparams[d.g_isl_world[i]];
        float4* dv = d.dv + kDvF4 * (size_t)bs;
        for (int k = 0; k < kDvF4 * bc; k++) dv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = rs; r < rs + rc; r++) row_warm(d.rows[r], d.rows[r].imp, dv);
        for (int it = 0; it < P.pgs_vel; it++)
            for (int r = rs; r < rs + rc; r++) {
                RowBlock& R = d.rows[r];
                float4 imp = R.imp;
                int st = R.stat;
                row_vel(R, imp, st, dv);
                R.imp = imp;
                R.stat = st;
            }
        for (int it = 0; it < P.pgs_pos; it++)
            for (int r = rs; r < rs + rc; r++) {
                RowBlock& R = d.rows[r];
                float4 imp = R.imp;
                row_pos(R, imp, dv);
                R.imp = imp;
            }
        island_finish(d, rs, rc, bs, bc, dv, 0, 1);
    }
}

// ---- large islands: one warp per island, rows streamed through shared memory
// 36 KB of rows per chain; chunks of 32 rows measured 279 cycles per row-step on
// a 2,000-row chain, of 16 rows 297 (the work at a chunk's edge)
constexpr int kRingSlots = 3;
constexpr int kChunkRows = 32;

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// `fence`: this thread wrote impulses to `src` with generic stores since its
// last proxy fence; those writes must be ordered before the async-proxy copy
// reads them.  (Its earlier reads of `dst` have completed: their values were
// used before this copy is issued.)
__device__ __forceinline__ void ring_load(RowBlock* dst, const RowBlock* src, int rows, uint64_t* bar, bool fence) {
    uint32_t bytes = (uint32_t)(rows * sizeof(RowBlock));
    if (fence) asm volatile("fence.proxy.async;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(saddr(dst)),
                 "l"(src), "r"(bytes), "r"(saddr(bar))
                 : "memory");
}

__device__ __forceinline__ bool ring_wait(uint64_t* bar, uint32_t parity, long long limit) {
    for (long long it = 0; it < limit; it++) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(saddr(bar)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// ---- the chain of one island on two lanes -------------------------------------
// Gauss-Seidel is serial, so a large island costs its row-steps one after the
// other.  On one lane a row-step issues ~150 instructions (~460 cycles; its
// dependency chain is ~130), so two lanes share it, one body of the contact
// each: a lane reads its body's half of the row (144 of 288 bytes), forms its
// three partial dot products, meets the other lane's by shuffle (the sum is
// the same either way round, so both get the bits of the one-lane row),
// evaluates the row's scalars alongside and updates its own body's Δv.  That
// halves the loads, dot products and updates, and leaves the registers to
// load the next row while the current one is solved.  A lane keeps its body
// while consecutive rows share it, whichever side of the row it is on; the Δv
// of a body that changes is read one row ahead.  A row's code has no branch but a
// uniform one for rows that slide (any other costs a lone warp ~40 cycles), and
// the whole warp runs it, even lanes
// as lane 0 and odd lanes as lane 1 (same addresses, same values): two lanes
// inside a branch would check for divergence at every shuffle (404 cycles per
// row-step against 307).  Measured on a chain of 2,000 rows: 459 -> 233 cycles
// per row-step where contacts stick, 252 with 28 % of them sliding, 304 where all
// slide; of 90 rows (held in shared memory) with 28 %: 523 -> 253.

struct HalfRow {
    float2 j[9];     // J of the normal and friction rows (u, w) for the lane's body, three component pairs each
    float2 m[9];     // M^-1 J^T of the same
    float4 imp;      // impulses: normal, pseudo normal, friction u, w
    float4 tgt;      // targets n, u, w; friction coefficient
    float4 nrm;      // nminv, nptarget, kd0, kd1
    float4 fm;       // Fm^-1 by columns
};
__device__ __forceinline__ void half_load(const RowBlock* R, int side, HalfRow& h) {
    const float4* q = reinterpret_cast<const float4*>(R);
    h.imp = q[0];
    h.tgt = q[3];
    h.nrm = q[4];
    h.fm = q[5];
    const float4* s = q + 6 + 9 * side;
    float2 f[18];
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const float4 x = s[k];
        f[2 * k] = make_float2(x.x, x.y);
        f[2 * k + 1] = make_float2(x.z, x.w);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) { h.j[k] = f[k]; h.m[k] = f[9 + k]; }
}
// one body's part of pdot
__device__ __forceinline__ float2 half_dot(const float2* j, const P3& v) {
    float2 s = __fmul2_rn(j[0], v.a);
    s = __ffma2_rn(j[1], v.b, s);
    return __ffma2_rn(j[2], v.c, s);
}
// ... and its sum with the other lane's part
__device__ __forceinline__ float2 half_other(float2 s) {
    return make_float2(__shfl_xor_sync(0xffffffffu, s.x, 1), __shfl_xor_sync(0xffffffffu, s.y, 1));
}
__device__ __forceinline__ float half_sum(float2 s, float2 o) {
    const float2 u = __fadd2_rn(s, o);
    return __fadd_rn(u.x, u.y);
}
__device__ __forceinline__ void half_axpy(P3& v, const float2* m, float s) {
    const float2 b = bc2(s);
    v.a = __ffma2_rn(m[0], b, v.a);
    v.b = __ffma2_rn(m[1], b, v.b);
    v.c = __ffma2_rn(m[2], b, v.c);
}
__device__ __forceinline__ P3 psel(bool first, const P3& x, const P3& y) {
    return P3{make_float2(first ? x.a.x : y.a.x, first ? x.a.y : y.a.y),
              make_float2(first ? x.b.x : y.b.x, first ? x.b.y : y.b.y),
              make_float2(first ? x.c.x : y.c.x, first ? x.c.y : y.c.y)};
}
template <bool SH>
__device__ __forceinline__ P3 dv_load(const float4* dv, int slot, int which) {
    return SH ? dv_get_z(dv, slot, which) : dv_get(dv, slot, which);
}
// the same by scalar FMAs: no broadcast of s into a register pair, which the
// chain would wait for
__device__ __forceinline__ void half_axpy1(P3& v, const float2* m, float s) {
    v.a = make_float2(__fmaf_rn(m[0].x, s, v.a.x), __fmaf_rn(m[0].y, s, v.a.y));
    v.b = make_float2(__fmaf_rn(m[1].x, s, v.b.x), __fmaf_rn(m[1].y, s, v.b.y));
    v.c = make_float2(__fmaf_rn(m[2].x, s, v.c.x), __fmaf_rn(m[2].y, s, v.c.y));
}
// row_warm for the lane's body
__device__ __forceinline__ void half_warm(const HalfRow& h, P3& v) {
    if (fabsf(h.imp.x) > kZero) half_axpy(v, h.m, h.imp.x);
    if (fabsf(h.imp.z) > kZero || fabsf(h.imp.w) > kZero) {
        half_axpy(v, h.m + 3, h.imp.z);
        half_axpy(v, h.m + 6, h.imp.w);
    }
}
// row_pos for the lane's body (pseudo velocities p)
__device__ __forceinline__ void half_pos(HalfRow& h, P3& p) {
    const float2 s = half_dot(h.j, p);
    const float cur = half_sum(s, half_other(s));
    const float nw = __fmaf_rn(h.nrm.x, __fsub_rn(h.nrm.y, cur), h.imp.y);
    const float diff = __fsub_rn(fmaxf(nw, 0.0f), h.imp.y);
    if (fabsf(diff) > kZero) {
        half_axpy(p, h.m, diff);
        h.imp.y = __fadd_rn(h.imp.y, diff);
    }
}
// row_vel_r for the lane's body
__device__ __forceinline__ void half_vel(HalfRow& h, P3& v, int& stat) {
    const float2 sn = half_dot(h.j, v), s0 = half_dot(h.j + 3, v), s1 = half_dot(h.j + 6, v);
    const float2 on = half_other(sn), o0 = half_other(s0), o1 = half_other(s1);
    const float cur = half_sum(sn, on), b0 = half_sum(s0, o0), b1 = half_sum(s1, o1);
    const float nw = __fmaf_rn(h.nrm.x, __fsub_rn(h.tgt.x, cur), h.imp.x);
    const float2 g = psub(make_float2(h.tgt.y, h.tgt.z), make_float2(b0, b1));
    const float2 A = __fadd2_rn(make_float2(h.imp.z, h.imp.w),
                                __ffma2_rn(make_float2(h.fm.z, h.fm.w), bc2(g.y),
                                           __fmul2_rn(make_float2(h.fm.x, h.fm.y), bc2(g.x))));
    float diff = __fsub_rn(fmaxf(nw, 0.0f), h.imp.x);
    if (!(fabsf(diff) > kZero)) diff = 0.f;
    const float ix = __fadd_rn(h.imp.x, diff);
    half_axpy(v, h.m, diff);
    float2 nf = __ffma2_rn(bc2(-diff), make_float2(h.nrm.z, h.nrm.w), A);
    const float mx = __fmul_rn(h.tgt.w, ix);
    const float s2 = __fmaf_rn(nf.x, nf.x, __fmul_rn(nf.y, nf.y));
    // The clamp's rsqrt is ~49 cycles of dependent work: the row goes on as if
    // it stuck, and is put right where it slides.  The vote makes that branch a
    // uniform one (a branch on a lane's own condition costs a lone warp ~40
    // cycles more).
    const float2 old = make_float2(h.imp.z, h.imp.w);
    const bool slide = s2 > __fmul_rn(mx, mx);
    float2 e = psub(nf, old);
    if (!(fabsf(e.x) > kZero || fabsf(e.y) > kZero)) e = make_float2(0.f, 0.f);
    P3 w = v;
    half_axpy1(w, h.m + 3, e.x);
    half_axpy1(w, h.m + 6, e.y);
    stat = 1;
    if (__any_sync(0xffffffffu, slide)) {
        stat = 0;
        nf = __fmul2_rn(nf, bc2(__fmul_rn(mx, rsqrtf(s2))));
        e = psub(nf, old);
        if (!(fabsf(e.x) > kZero || fabsf(e.y) > kZero)) e = make_float2(0.f, 0.f);
        w = v;
        half_axpy1(w, h.m + 3, e.x);
        half_axpy1(w, h.m + 6, e.y);
    }
    v = w;
    h.imp.x = ix;
    h.imp.z = __fadd_rn(h.imp.z, e.x);
    h.imp.w = __fadd_rn(h.imp.w, e.y);
}

// A chain's rows in shared memory.  An island of at most kRingSlots chunks is
// resident: every chunk is copied in once and the passes run over it in
// place, impulses included.  A larger one streams through the ring, chunk c
// of a pass at sequence t = pass * chunks + c, looked ahead by at most one
// pass (a pass must see the impulses the previous pass wrote back).
struct RowFeed {
    RowBlock* ring;
    uint64_t* bars;
    RowBlock* rows;        // the island's rows in global memory
    uint32_t phase;        // bit k: parity of slot k
    int rc, nch, total, ahead;
    int t, slot;           // the chunk being read: sequence, ring slot
    int issued, islot, ic; // the next chunk to copy: sequence, ring slot, chunk index
    int fenced;            // sequence of the last proxy fence
    int first_write;       // sequence from which passes write impulses back
    bool lead;
    long long limit;

    // Copies the next chunk; the rows up to sequence `now` have been written
    // back.  A proxy fence covers every impulse write issued before it; the
    // chunk was last written at sequence issued - nch, so a fence is needed
    // only if none was issued since: about once per pass on a large island.
    __device__ __forceinline__ void issue(int now) {
        const int tw = issued - nch;
        const bool fence = tw >= first_write && tw > fenced;
        if (fence) fenced = now;
        if (lead)
            ring_load(ring + islot * kChunkRows, rows + ic * kChunkRows, min(kChunkRows, rc - ic * kChunkRows), &bars[islot], fence);
        issued++;
        if (++islot == kRingSlots) islot = 0;
        if (++ic == nch) ic = 0;
    }
    // the rows of the chunk at sequence t are in shared memory
    __device__ __forceinline__ bool arrive() {
        if (!ring_wait(&bars[slot], (phase >> slot) & 1u, limit)) {
            // gave up on chunk t: let the copies in flight land before the
            // ring is abandoned (bounded)
            for (int u = t; u < issued; u++) {
                ring_wait(&bars[slot], (phase >> slot) & 1u, kDefaultWaitLimit);
                if (++slot == kRingSlots) slot = 0;
            }
            return false;
        }
        phase ^= 1u << slot;
        return true;
    }
    __device__ __forceinline__ void advance() {
        t++;
        if (++slot == kRingSlots) slot = 0;
    }
    __device__ __forceinline__ RowBlock* rows_at() const { return ring + slot * kChunkRows; }
    // the rows of the chunks up to sequence t - 1 have been read and their
    // impulses written: refill their slots
    __device__ __forceinline__ void refill() {
        while (issued < total && issued < t + ahead) issue(t - 1);
    }
};

// A run of n consecutive rows at `row` (shared memory), in order; KIND 0: warm
// start, with the first position pass fused in when there is one (the position
// rows read and write only the pseudo velocities and the pseudo impulse, which
// no other pass touches and which start at zero, so position row j right after
// warm-start row j gives the same result as a separate pass, one pass sooner);
// 1: a velocity pass; 3: the last one (the friction state is stored too); 2: a
// position pass.  The first row is already in `A`; each row's successor (`then`
// after the last one) is loaded while the row is solved, without a branch in a
// row's code.  Impulses go to `out`; `fin`: also there (KIND 3).
// SH: `dv` is in shared memory with a zero entry at index -1 for the bodies of
// infinite mass.  The entry is never written and every row reads it anew: M^-1 J^T
// is zero there, but zero times an overflowing impulse is NaN, and the entry
// serves every island of the worker.
struct ChainState {
    P3 v, p;       // Δv and pseudo Δv of the lane's body
    int own;       // its slot
    int side;      // the side of the row it is on
    int sa, sb;    // the row's slots
};
template <int KIND, bool SH, bool FUSED>
__device__ __forceinline__ void chain_run(const RowBlock* row, int n, const RowBlock* then, RowBlock* out, RowBlock* fin, float4* dv,
                                          ChainState& c, HalfRow& A) {
    constexpr bool kV = KIND != 2, kP = KIND == 2 || (KIND == 0 && FUSED);
    int left = n;
    auto step = [&](HalfRow& cur, HalfRow& nxt) {
        left--;
        const RowBlock* next = left == 0 ? then : row + 1;
        const int na = next->sa, nb = next->sb;
        // a body that changes sides stays with its lane
        const int nside = c.side ^ (int)((na == c.sb) | (nb == c.sa));
        const int nown = nside ? nb : na;
        half_load(next, nside, nxt);
        P3 nv{}, np{};
        if (kV) nv = dv_load<SH>(dv, nown, 0);
        if (kP) np = dv_load<SH>(dv, nown, 1);
        int stat = 0;
        if (KIND == 0) {
            half_warm(cur, c.v);
            if (FUSED) half_pos(cur, c.p);
        } else if (KIND == 2) {
            half_pos(cur, c.p);
        } else {
            half_vel(cur, c.v, stat);
        }
        if (KIND != 0 || FUSED) {   // both lanes, the same value
            out->imp = cur.imp;
            if (KIND == 3) {
                fin->imp = cur.imp;
                fin->stat = stat;
                fin++;
            }
            out++;
        }
        if (kV) dv_put(dv, c.own, 0, c.v);
        if (kP) dv_put(dv, c.own, 1, c.p);
        __syncwarp(0xffffffffu);   // the other lane may read this body next
        const bool keep = nown == c.own && nown >= 0;
        if (kV) c.v = psel(keep, c.v, nv);
        if (kP) c.p = psel(keep, c.p, np);
        c.own = nown;
        c.side = nside;
        c.sa = na;
        c.sb = nb;
        row = next;
    };
    HalfRow B;
    while (left > 1) {
        step(A, B);
        step(B, A);
    }
    if (left) step(A, B);
}

// One pass over the island's rows.  RES: the rows are resident (one run in
// place, impulses included); otherwise a run per chunk, the next chunk's
// arrival waited for before the run that looks ahead to it.
template <int KIND, bool SH, bool RES, bool FUSED>
__device__ __forceinline__ bool chain_pass(RowFeed& x, float4* dv, int lane) {
    constexpr bool kV = KIND != 2, kP = KIND == 2 || (KIND == 0 && FUSED);
    if (!RES) {
        x.refill();
        if (!x.arrive()) return false;
    }
    RowBlock* row = RES ? x.ring : x.rows_at();
    ChainState c{};
    c.sa = row->sa;
    c.sb = row->sb;
    c.side = lane;
    c.own = lane ? c.sb : c.sa;
    if (kV) c.v = dv_load<SH>(dv, c.own, 0);
    if (kP) c.p = dv_load<SH>(dv, c.own, 1);
    HalfRow A;
    half_load(row, lane, A);
    if (RES) {
        chain_run<KIND, SH, FUSED>(row, x.rc, row, row, x.rows, dv, c, A);
    } else {
        RowBlock* out = x.rows;
        for (int k = 0; k < x.nch; k++) {
            const int n = min(kChunkRows, x.rc - k * kChunkRows);
            RowBlock* then = row;
            x.refill();
            x.advance();
            if (k + 1 < x.nch) {
                if (!x.arrive()) return false;
                then = x.rows_at();
            }
            chain_run<KIND, SH, FUSED>(row, n, then, out, out, dv, c, A);
            row = then;
            out += n;
        }
    }
    return true;
}

// the chain of one island: 1 warm-start pass, pgs_vel velocity passes and
// pgs_pos position passes over its rows
template <bool SH, bool RES>
__device__ __forceinline__ bool chain_passes(RowFeed& x, float4* dv, int lane, int n_vel, int n_pos) {
    if (RES)
        while (x.t < x.total) {
            if (!x.arrive()) return false;
            x.advance();
        }
    bool ok = n_pos > 0 ? chain_pass<0, SH, RES, true>(x, dv, lane & 1) : chain_pass<0, SH, RES, false>(x, dv, lane & 1);
    for (int k = 1; ok && k < n_vel; k++) ok = chain_pass<1, SH, RES, false>(x, dv, lane & 1);
    if (ok && n_vel > 0) ok = chain_pass<3, SH, RES, false>(x, dv, lane & 1);
    for (int k = 1; ok && k < n_pos; k++) ok = chain_pass<2, SH, RES, false>(x, dv, lane & 1);
    return ok;
}
template <bool SH>
__device__ __forceinline__ bool big_chain(const Dev& d, RowBlock* ring, uint64_t* bars, uint32_t& phase, float4* dv, int rs,
                                       int rc, const WorldParams& P, int lane) {
    const int n_vel = P.pgs_vel;   // read once: the row stores could alias P for the compiler
    const int n_pos = P.pgs_pos;
    const bool fused = n_pos > 0;
    const int passes = 1 + n_vel + (fused ? n_pos - 1 : 0);
    RowFeed x;
    x.ring = ring;
    x.bars = bars;
    x.rows = d.rows + rs;
    x.phase = phase;
    x.rc = rc;
    x.nch = (rc + kChunkRows - 1) / kChunkRows;
    const bool resident = x.nch <= kRingSlots;
    x.total = resident ? x.nch : passes * x.nch;
    x.ahead = x.nch < kRingSlots ? x.nch : kRingSlots;
    x.t = x.slot = x.issued = x.islot = x.ic = 0;
    x.fenced = -1;
    x.first_write = fused ? 0 : x.nch;
    x.lead = lane == 0;
    x.limit = d.wait_limit;
    // the previous island may have written the ring in place
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp(0xffffffffu);
    x.refill();
    const bool ok = resident ? chain_passes<SH, true>(x, dv, lane, n_vel, n_pos) : chain_passes<SH, false>(x, dv, lane, n_vel, n_pos);
    phase = x.phase;
    return ok;
}

// One warp's solver-chain worker: takes the big-island list's entries through
// `counter` and runs the chains of its islands -- SH: those of at most `dv_cap`
// bodies, whose Δv stays in shared memory; otherwise the larger ones, Δv in
// global memory.  `sm`: the warp's own shared area (mbarriers, row ring, the
// zero entry of the bodies of infinite mass, Δv).  A bounded wait that gives
// up ends the worker (the status is set).
template <bool SH>
__device__ void big_worker(const Dev& d, int dv_cap, uint8_t* sm, int* counter, int n) {
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm);
    RowBlock* ring = reinterpret_cast<RowBlock*>(sm + 64);
    float4* sdv = reinterpret_cast<float4*>(sm + 64 + kRingSlots * kChunkRows * sizeof(RowBlock)) + kDvF4;
    const int lane = threadIdx.x & 31;
    if (lane == 0)
        for (int k = 0; k < kRingSlots; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(&bars[k])), "r"(1) : "memory");
        }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (SH && lane < kDvF4) sdv[lane - kDvF4] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    uint32_t phase = 0;   // bit k: parity of slot k
    while (true) {
        int q = 0;
        if (lane == 0) q = atomicAdd(counter, 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= n) break;
        const int i = d.big_list[q];
        const int bs = d.g_isl_body_start[i], bc = d.g_isl_body_count[i];
        if (SH != (bc <= dv_cap)) continue;
        const int rs = d.g_isl_row_start[i], rc = d.g_isl_row_count[i];
        const WorldParams& P = d.wparams[d.g_isl_world[i]];
        float4* dv = SH ? sdv : d.dv + kDvF4 * (size_t)bs;
        for (int k = lane; k < kDvF4 * bc; k += 32) dv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
        bool ok = big_chain<SH>(d, ring, bars, phase, dv, rs, rc, P, lane);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
            if (lane == 0) atomicOr(d.status, ST_TIMEOUT);
            return;
        }
        __syncwarp();
        island_finish(d, rs, rc, bs, bc, dv, lane, 32);
        __syncwarp();
    }
}

// sched[kBigNext + (SH ? 0 : 1)]: the next list entry
constexpr int kBigNext = 8;

// blockDim.x == 32; `dv_cap` island bodies fit in the shared Δv area
template <bool SH>
__global__ void __launch_bounds__(32) k_pgs_big(Dev d, int dv_cap) {
    extern __shared__ __align__(16) uint8_t sm[];
    big_worker<SH>(d, dv_cap, sm, &d.sched[kBigNext + (SH ? 0 : 1)], d.sched[0]);
}

// Islands of a few rows: the chain with all of the island's rows in shared
// memory, 21 KB a warp, so that many run beside each other (the big islands'
// workers take two to five to an SM).  A thread walking its rows in global
// memory takes 0.2 to 0.45 us a row-step against 0.13 here, but a warp's start
// and end cost ~4 us an island: from 4 rows while one or a few islands fall to a
// warp, from 16 in batches of more islands.  Beside a chain of 512 rows or more,
// which bounds the step, only `few` blocks run (the others would hold shared
// memory that the big islands' workers need).
constexpr int kMidSmem = 64 + kMidMax * (int)sizeof(RowBlock) + (kMidMax + 2) * 16 * kDvF4;
constexpr int kMidNext = kBigNext + 3;   // sched: the next list entry
__global__ void __launch_bounds__(32) k_pgs_mid(Dev d, int few) {
    extern __shared__ __align__(16) uint8_t sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    RowBlock* ring = reinterpret_cast<RowBlock*>(sm + 64);
    float4* dv = reinterpret_cast<float4*>(sm + 64 + kMidMax * sizeof(RowBlock)) + kDvF4;   // after the zero entry
    if ((int)blockIdx.x >= few && d.sched[kLongIslands] > 0) return;
    const int lane = threadIdx.x, n = d.sched[kMidIslands];
    if ((int)blockIdx.x >= n) return;
    if (lane == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (lane < kDvF4) dv[lane - kDvF4] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    uint32_t parity = 0;
    while (true) {
        int q = 0;
        if (lane == 0) q = atomicAdd(&d.sched[kMidNext], 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= n) break;
        const int i = d.big_list[d.n_bodies - 1 - q];
        const int bs = d.g_isl_body_start[i], bc = d.g_isl_body_count[i];   // at most kMidMax + 1 bodies
        const int rs = d.g_isl_row_start[i], rc = d.g_isl_row_count[i];
        const WorldParams& P = d.wparams[d.g_isl_world[i]];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the last island's rows were written in place
        __syncwarp();
        if (lane == 0) ring_load(ring, d.rows + rs, rc, bar, false);
        for (int k = lane; k < kDvF4 * bc; k += 32) dv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int n_vel = P.pgs_vel, n_pos = P.pgs_pos;
        const bool ok = ring_wait(bar, parity, d.wait_limit);
        parity ^= 1u;
        if (!__all_sync(0xffffffffu, ok)) {
            ring_wait(bar, parity ^ 1u, kDefaultWaitLimit);   // let the copy land (bounded)
            if (lane == 0) atomicOr(d.status, ST_TIMEOUT);
            return;
        }
        RowFeed x;
        x.ring = ring;
        x.rows = d.rows + rs;
        x.rc = rc;
        x.t = x.total = 0;   // nothing left to arrive
        chain_passes<true, true>(x, dv, lane, n_vel, n_pos);
        __syncwarp();
        island_finish(d, rs, rc, bs, bc, dv, lane, 32);
        __syncwarp();
    }
}

// HolonomicSystem::computeAndApplyImpulses (HolonomicBlockSolver.cpp:319-378)
// for system s by one warp: solve A d = t - J dv with the factorisation, then
// (with a threshold) discard a pseudo solution whose angular velocity change
// exceeds it anywhere, else apply d.  `v`: the solve's vector; row(i): the
// staged part of constraint i's row.
template <class T, class Row>
__device__ __forceinline__ void holo_apply(const Dev& d, int s, const HoloView& h, T* v, const Row& row_of, float4* dv, float4* err,
                                           bool pseudo, float thr, int lane) {
    const HoloStore& hs = d.hs;
    const T* B = reinterpret_cast<const T*>(hs.fp64[s] ? (const void*)(hs.pool64 + hs.bstart[s])
                                                       : (const void*)(hs.pool32 + hs.bstart[s]));
    const int which = pseudo ? 1 : 0, n = h.n;
    for (int i = lane; i < n; i += 32) {
        const JointRow& R = *row_of(i);
        float va[6], vb[6], cur[kJMax];
        jload(dv, R.sa, which, va);
        jload(dv, R.sb, which, vb);
        jvalue(R, va, vb, cur);
        const float* tgt = pseudo ? R.ptarget : R.target;
        for (int k = 0; k < R.n; k++) v[h.vpos[i] + k] = (T)tgt[k] - (T)cur[k];
    }
    __syncwarp();
    holo_solve<T>(h, hs.table + hs.tstart[s], B, v, lane);
    // the solution's change of Δv, constraint by constraint in order (bodies
    // are shared); the next constraint's row is loaded meanwhile
    auto apply = [&](float4* to, int wh, bool store) {
        JointLane L, N;
        float imp = 0.f, nimp = 0.f;
        auto load = [&](int i, JointLane& x, float& z) {
            jl_load(*row_of(i), lane, x);
            z = lane < x.n ? (float)v[h.vpos[i] + lane] : 0.f;
        };
        load(0, L, imp);
        for (int i = 0; i < n; i++) {
            if (i + 1 < n) load(i + 1, N, nimp);
            if (__any_sync(0xffffffffu, fabsf(imp) > kJZero)) {
                jl_apply(L, imp, to, wh, lane);
                if (store && lane < L.n) {
                    JointRow& R = *row_of(i);
                    (pseudo ? R.pimpulse : R.holo)[lane] += imp;
                }
            }
            L = N;
            imp = nimp;
        }
        __syncwarp();
    };
    if (thr > 0.f) {
        apply(err, 0, false);
        bool over = false;
        for (int i = lane; i < n; i += 32) {
            const JointRow& R = *row_of(i);
            float ea[6], eb[6];
            jload(err, R.sa, 0, ea);
            jload(err, R.sb, 0, eb);
            float r2 = 0.f;
            for (int k = 3; k < 6; k++) r2 += ea[k] * ea[k] + eb[k] * eb[k];
            over = over || r2 > thr * thr;
        }
        if (__any_sync(0xffffffffu, over)) return;
    }
    apply(dv, which, true);
}

// a system's tables in shared memory: up to kHoloN constraints, kHoloL blocks
// below the diagonal
constexpr int kHoloN = 64, kHoloL = 96;
struct HoloSm {
    double v[kHoloN * kJMax + kJMax];
    int cons[kHoloN], vpos[kHoloN], dim[kHoloN], ls[kHoloN + 1], lrow[kHoloL], lloc[kHoloL];
    JointRow* rows[kHoloN];
};
// both solves of system s; res: find(j) gives joint j's row in shared memory or null
template <class T, class Find>
__device__ __noinline__ void holo_system(const Dev& d, int s, HoloSm& sm, bool res, const Find find, float4* dv, float4* err, int lane) {
    const HoloStore& hs = d.hs;
    const int c0 = hs.cstart[s], n = hs.cstart[s + 1] - c0;
    const int* ls = hs.lstart + hs.lbase[s];
    const int l0 = ls[0], nl = ls[n] - l0;
    T* work = reinterpret_cast<T*>(hs.work + hs.wstart[s]);
    if (n <= kHoloN && nl <= kHoloL) {
        for (int i = lane; i < n; i += 32) {
            const int j = hs.cons[c0 + i];
            sm.cons[i] = j;
            sm.vpos[i] = hs.vpos[c0 + i];
            sm.dim[i] = d.jt.rows[j].n;
            JointRow* r = res ? find(j) : nullptr;
            sm.rows[i] = r ? r : d.jt.rows + j;
        }
        for (int i = lane; i <= n; i += 32) sm.ls[i] = ls[i];
        for (int i = lane; i < nl; i += 32) { sm.lrow[i] = hs.lrow[l0 + i]; sm.lloc[i] = hs.lloc[l0 + i]; }
        __syncwarp();
        const HoloView h{n, sm.cons, sm.vpos, sm.ls, sm.lrow, sm.lloc, sm.dim, l0};
        auto row = [&](int i) { return sm.rows[i]; };
        for (int p = 0; p < 2; p++)
            holo_apply<T>(d, s, h, reinterpret_cast<T*>(sm.v), row, dv, err, p == 1, p == 1 ? d.lin_err_threshold : -1.f, lane);
        __syncwarp();
    } else {
        const HoloView h{n, hs.cons + c0, hs.vpos + c0, ls, hs.lrow, hs.lloc, hs.dim + c0, 0};
        auto row = [&](int i) { return d.jt.rows + h.cons[i]; };
        for (int p = 0; p < 2; p++)
            holo_apply<T>(d, s, h, work, row, dv, err, p == 1, p == 1 ? d.lin_err_threshold : -1.f, lane);
    }
}

// A joint-island warp's shared memory (k_pgs_joint): what is held and up to which
// island (more in global memory).
constexpr int kJointDv = 68, kJointRes = 64, kJointList = 1024;
constexpr int kRowF4 = (int)(sizeof(RowBlock) / 16);
struct alignas(16) JointSm {
    uint64_t bar;
    float zero[8];              // Δv of a body of infinite mass
    int held[kJointRes];        // the joint in each slot
    int16_t list[kJointList];   // the row's joint slot, -1 a contact row
    HoloSm holo;
    float4 crow[2][kRowF4];     // contact rows on their way to the lanes
    float4 dv[kDvF4 * kJointDv];
    uint8_t rows[kJointRes * kJointStage];
};
constexpr int kJointSmem = (int)sizeof(JointSm);
static_assert(offsetof(JointSm, rows) % 16 == 0 && kJointStage % 16 == 0, "bulk copies into the held rows");
__device__ __forceinline__ JointSm& joint_sm() {
    extern __shared__ __align__(16) uint8_t sm[];
    return *reinterpret_cast<JointSm*>(sm);
}

// The passes over a joint island's rows.  A joint row takes the lanes of joints.cuh
// with only the pass's own fields loaded and, where the island is held in shared
// memory, everything typed as such: it is bound by its instruction count on one
// warp (168 a row-step through generic pointers) and its dependency chain.  A
// step is PGSConstraintStep<n> (ConstraintSolver.cpp:12-40): the accumulated impulse
// plus the row's correction, projected (ConeLimitConstraint /
// TwistLimitConstraint::projectValidImpulse, ConstraintSolver.cpp:434-436,
// 463-465: one-sided limits; MotorConstraint / PistonConstraint, :591-606,
// 728-731), applied when the change is not zero.  A contact row is shared by two
// lanes like the large islands' (half_vel and the others above; by lane 0 alone,
// from global memory: 32 chains of 30 links lying on a plate 5.6 ms a step, now 3.5).
struct JointRes {
    int n, sa, sb, proj, pos;
    float lim, ja[6], jb[6], mv[6], it[6], tgt, acc;
};
template <int KIND>
__device__ __forceinline__ void jr_load(const uint8_t* row, int lane, JointRes& L) {
    const JointRow& R = *reinterpret_cast<const JointRow*>(row);
    const int i = min(lane, 5), c = min(lane, 11);
    const int4 h = *reinterpret_cast<const int4*>(&R.n);
    L.n = h.x; L.sa = h.y; L.sb = h.z; L.proj = h.w;
    jl_row6(R.ita + kJMax * c, L.it);   // body b's follow body a's
    if (KIND == 0) {
        L.acc = R.impulse[i];
        return;
    }
    L.lim = R.lim;
    L.pos = R.pos;
    jl_row6(R.ja + 6 * i, L.ja);
    jl_row6(R.jb + 6 * i, L.jb);
    jl_row6(R.minv + kJMax * i, L.mv);
    L.tgt = KIND == 1 ? R.target[i] : R.ptarget[i];
    L.acc = KIND == 1 ? R.impulse[i] : R.pimpulse[i];
}
__device__ __forceinline__ const float* jr_dv(const float4* dv, const float* zero, int slot, int which) {
    return slot < 0 ? zero : reinterpret_cast<const float*>(dv + kDvF4 * slot) + 6 * which;
}
template <int KIND>
__device__ __forceinline__ void jr_row(const JointRes& L, uint8_t* row, float4* dv, const float* zero, int lane) {
    constexpr int which = KIND == 2 ? 1 : 0;
    if (KIND == 2 && !L.pos) return;   // needsPosCorrect
    const int slot = lane < 6 ? L.sa : L.sb, comp = lane < 6 ? lane : min(lane, 11) - 6;
    const float old = jr_dv(dv, zero, slot, which)[comp];
    float imp;
    if (KIND == 0) {
        imp = L.acc;
    } else {
        float va[6], vb[6];
        jl_row6(jr_dv(dv, zero, L.sa, which), va);
        jl_row6(jr_dv(dv, zero, L.sb, which), vb);
        float x = 0.f, y = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            x = __fmaf_rn(va[k], L.ja[k], x);
            y = __fmaf_rn(vb[k], L.jb[k], y);
        }
        const float delta = __fsub_rn(L.tgt, __fadd_rn(x, y));
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) s = __fmaf_rn(__shfl_sync(0xffffffffu, delta, k), L.mv[k], s);
        float nw = __fadd_rn(L.acc, s);
        if (__any_sync(0xffffffffu, L.proj != 0)) {   // rows of one dof
            if (L.proj == 1) nw = fmaxf(nw, 0.f);
            else if (L.proj == 2) nw = fminf(nw, 0.f);
            else nw = nw > 0.f ? fminf(nw, L.lim) : fmaxf(nw, -L.lim);
        }
        imp = __fsub_rn(nw, L.acc);
        if (lane >= L.n) imp = 0.f;   // a projection's value beyond the row's one dof
    }
    if (__any_sync(0xffffffffu, fabsf(imp) > kJZero)) {
        float x = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) x = __fmaf_rn(__shfl_sync(0xffffffffu, imp, k), L.it[k], x);
        if (lane < 12 && slot >= 0) const_cast<float*>(jr_dv(dv, zero, slot, which))[comp] = __fadd_rn(old, x);
        if (KIND != 0 && lane < L.n) {
            JointRow& R = *reinterpret_cast<JointRow*>(row);
            (KIND == 1 ? R.impulse : R.pimpulse)[lane] = __fadd_rn(L.acc, imp);
        }
    }
    __syncwarp();
}
// a contact row in shared memory at `sr`, its own place `R`
template <int KIND>
__device__ __forceinline__ void jc_row(const RowBlock* sr, RowBlock* R, float4* dv, int lane) {
    constexpr int which = KIND == 2 ? 1 : 0;
    HalfRow h;
    half_load(sr, lane & 1, h);
    const int slot = lane & 1 ? sr->sb : sr->sa;
    P3 v = dv_get(dv, slot, which);
    int stat = 0;
    if (KIND == 0) half_warm(h, v);
    else if (KIND == 1) half_vel(h, v, stat);
    else half_pos(h, v);
    if (KIND != 0) R->imp = h.imp;   // all lanes, the same value
    if (KIND == 1) R->stat = stat;
    dv_put(dv, slot, which, v);
    __syncwarp();
}
// One pass.  KIND 0: warm start, 1: velocity, 2: position.  RES: joint rows and Δv
// are in shared memory; MIXED: the island holds contact rows.  The next contact
// row is loaded by 24 lanes, 16 bytes each, and goes through shared memory.
template <int KIND, bool RES, bool MIXED>
__device__ __forceinline__ void joint_pass(JointSm& sm, JointRow* joints, RowBlock* rows, int rc, float4* dv, int lane) {
    JointRes A, B;
    float4 piece{};
    const float* zero = sm.zero;
    // row r's joint slot (RES) or joint, -1 a contact row
    auto kind = [&](int r) {
        if (RES) return (int)sm.list[r];
        const int c = rows[r].contact;
        return c < 0 ? -c - 1 : -1;
    };
    auto joint = [&](int k) { return RES ? sm.rows + k * kJointStage : reinterpret_cast<uint8_t*>(joints + k); };
    auto load = [&](int k, int at, JointRes& J) {
        jr_load<KIND>(joint(max(k, 0)), lane, J);   // without a branch: some joint's in the place of a contact row
        if (MIXED) piece = reinterpret_cast<const float4*>(rows + at)[min(lane, kRowF4 - 1)];
    };
    int c = kind(0), n = kind(min(1, rc - 1)), r = 0;
    load(c, 0, A);
    auto one = [&](JointRes& L, JointRes& N) {
        float4* sr = sm.crow[r & 1];
        if (MIXED && lane < kRowF4) sr[lane] = piece;
        load(n, min(r + 1, rc - 1), N);
        const int n2 = kind(min(r + 2, rc - 1));
        if (!MIXED || __any_sync(0xffffffffu, c >= 0)) {   // a vote: a uniform branch
            jr_row<KIND>(L, joint(c), dv, zero, lane);
        } else {
            __syncwarp();
            jc_row<KIND>(reinterpret_cast<const RowBlock*>(sr), rows + r, dv, lane);
        }
        c = n;
        n = n2;
        r++;
    };
    while (true) {
        one(A, B);
        if (r >= rc) break;
        one(B, A);
        if (r >= rc) break;
    }
    __syncwarp();
}
// the island's passes; a function of its own for the registers (inlined three
// times into the kernel they spilled)
template <bool RES, bool MIXED>
__device__ __forceinline__ void joint_passes(JointRow* joints, RowBlock* rows, int rc, float4* gdv, int n_vel, int n_pos, int lane) {
    JointSm& sm = joint_sm();
    float4* dv = RES ? sm.dv : gdv;
    joint_pass<0, RES, MIXED>(sm, joints, rows, rc, dv, lane);
    for (int it = 0; it < n_vel; it++) joint_pass<1, RES, MIXED>(sm, joints, rows, rc, dv, lane);
    for (int it = 0; it < n_pos; it++) joint_pass<2, RES, MIXED>(sm, joints, rows, rc, dv, lane);
}

// Islands with joint rows: one warp per island, contact rows and joint rows in
// island order, then the island's holonomic systems (first substep).  Bound by the
// chain of row-steps, each a few dependent loads: the joint rows (up to kJointRes
// of an island of up to kJointList rows) and the Δv of islands of up to kJointDv
// bodies (`dv_cap` lowers it) are held in shared memory.  On 512 chains of 16-64
// links: one lane and everything in global memory 568 us a substep, the rows
// in global memory 263, in shared memory 219, with each pass's own fields alone
// 131 (the first, with the solve, 1,880 -> 594 -> 438).  Past the lines (and past those of the block solve: kHoloN, kHoloL and
// the factor's kFactorBytes), a step of 256 hung chains of 64 / 65 / 69 / 100
// links, FP64 systems: 1.98 / 3.17 / 4.31 / 6.61 ms (6.78 / 6.84 / 7.64 / 12.8 by
// one lane with everything in global memory).
// sched[kJointNext]: the next joint-list entry
constexpr int kJointNext = kBigNext + 2;
__global__ void __launch_bounds__(32, 3) k_pgs_joint(Dev d, int first, int dv_cap) {
    JointSm& sm = joint_sm();
    uint64_t* bar = &sm.bar;
    int* held_j = sm.held;
    int16_t* list = sm.list;
    float4* sdv = sm.dv;
    uint8_t* srows = sm.rows;
    const int lane = threadIdx.x;
    const int nj = d.sched[3];
    uint32_t parity = 0;
    if (lane == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (lane < 8) sm.zero[lane] = 0.f;
    __syncwarp();
    while (true) {
        int q = 0;
        if (lane == 0) q = atomicAdd(&d.sched[kJointNext], 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= nj) break;
        const int i = d.joint_list[q];
        const int rs = d.g_isl_row_start[i], rc = d.g_isl_row_count[i];
        const int bs = d.g_isl_body_start[i], bc = d.g_isl_body_count[i];
        const WorldParams& P = d.wparams[d.g_isl_world[i]];
        float4* dv = bc <= dv_cap ? sdv : d.dv + kDvF4 * (size_t)bs;
        float4* err = d.dv_err + kDvF4 * (size_t)bs;
        // the island's joint rows into shared memory, if they fit
        int held = 0;
        bool res = rc <= kJointList && bc <= dv_cap;
        for (int base = 0; res && base < rc; base += 32) {
            const bool in = base + lane < rc;
            const int c = in ? d.rows[rs + base + lane].contact : 0;
            const unsigned m = __ballot_sync(0xffffffffu, c < 0);
            const int slot = held + __popc(m & ((1u << lane) - 1u));
            if (in) {
                list[base + lane] = c < 0 ? (int16_t)slot : (int16_t)-1;
                if (c < 0 && slot < kJointRes) held_j[slot] = -c - 1;
            }
            held += __popc(m);
            res = held <= kJointRes;
        }
        if (res && held > 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the last island's rows were written in place
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"((uint32_t)(held * kJointStage))
                             : "memory");
            __syncwarp();
            for (int r = lane; r < rc; r += 32)
                if (list[r] >= 0)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                     saddr(srows + list[r] * kJointStage)),
                                 "l"(d.jt.rows + (-d.rows[rs + r].contact - 1)), "r"((uint32_t)kJointStage), "r"(saddr(bar))
                                 : "memory");
        }
        for (int k = lane; k < kDvF4 * bc; k += 32) { dv[k] = make_float4(0.f, 0.f, 0.f, 0.f); err[k] = dv[k]; }
        __syncwarp();
        if (res && held > 0) {
            const bool ok = ring_wait(bar, parity, d.wait_limit);
            parity ^= 1u;
            if (!__all_sync(0xffffffffu, ok)) {
                ring_wait(bar, parity ^ 1u, kDefaultWaitLimit);   // let the copies in flight land (bounded)
                if (lane == 0) atomicOr(d.status, ST_TIMEOUT);
                return;
            }
        }
        const int n_vel = P.pgs_vel, n_pos = P.pgs_pos;   // read once: the row stores could alias P
        if (res && held == rc) joint_passes<true, false>(d.jt.rows, d.rows + rs, rc, dv, n_vel, n_pos, lane);
        else if (res) joint_passes<true, true>(d.jt.rows, d.rows + rs, rc, dv, n_vel, n_pos, lane);
        else joint_passes<false, true>(d.jt.rows, d.rows + rs, rc, dv, n_vel, n_pos, lane);
        if (first && P.pgs_holo > 0) {
            const int ss = d.g_isl_sys_start[i], sn = d.g_isl_sys_count[i];
            for (int it = 0; it < P.pgs_holo; it++)
                for (int k = 0; k < sn; k++) {
                    const int s = d.isl_sys[ss + k];
                    auto find = [=](int j) -> JointRow* {
                        for (int q = 0; q < held; q++)
                            if (held_j[q] == j) return reinterpret_cast<JointRow*>(srows + q * kJointStage);
                        return nullptr;
                    };
                    if (d.hs.fp64[s]) holo_system<double>(d, s, sm.holo, res, find, dv, err, lane);
                    else holo_system<float>(d, s, sm.holo, res, find, dv, err, lane);
                }
        }
        __syncwarp();
        for (int r = rs + lane; r < rs + rc; r += 32) {
            const int c = d.rows[r].contact;
            if (c >= 0) continue;
            const int j = -c - 1;
            const JointRow& R = res ? *reinterpret_cast<const JointRow*>(srows + list[r - rs] * kJointStage) : d.jt.rows[j];
            for (int k = 0; k < R.n; k++) {
                d.jt.impulse[kJMax * j + k] = R.impulse[k];
                if (res) {   // a row that is kept (a limit, a motor) goes on from these
                    d.jt.rows[j].impulse[k] = R.impulse[k];
                    d.jt.rows[j].pimpulse[k] = R.pimpulse[k];
                    d.jt.rows[j].holo[k] = R.holo[k];
                }
            }
        }
        island_finish(d, rs, rc, bs, bc, dv, lane, 32);
        __syncwarp();
    }
}

__device__ M33 crossm(f3 v) {
    M33 o;
    o.m[0] = 0.f;  o.m[1] = -v.z; o.m[2] = v.y;
    o.m[3] = v.z;  o.m[4] = 0.f;  o.m[5] = -v.x;
    o.m[6] = -v.y; o.m[7] = v.x;  o.m[8] = 0.f;
    return o;
}

__global__ void k_integrate(Dev d, int last) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_bodies; i += gridDim.x * blockDim.x) {
        const int mv = d.movement[i];
        if (mv == 1 || (d.has_sleep && d.asleep[i])) continue;   // sleeping bodies stay put
        const WorldParams& P = d.wparams[d.world[i]];
        const float dt = P.dt_sub;
        float4 pos = d.pos[i], q = d.rot[i];
        const float4 pos0 = pos, q0 = q;
        f3 v = mk(d.vel[i]), w = mk(d.angv[i]), pv = mk(d.pvel[i]), pw = mk(d.pangv[i]);
        f3 c = mk(pos) + (v + pv) * dt;
        pos.x = c.x; pos.y = c.y; pos.z = c.z;
        if (mag2(w) != 0.f) {
            const bool no_gyro = P.gyro_disabled || mv == 2;
            if (no_gyro) {
                q = qmul(qaxis(mag(w) * dt, normalize(w)), q);
            } else {
                // RigidBody::rotateWhileApplyingGyroAccel: implicit Euler on the
                // gyroscopic term, angle_ticks sub-steps of two Newton iterations
                const M33 Iref = load9(d.iref + 9 * i);
                M33 it = load9(d.iw + 9 * i);
                float4 iq = q;
                f3 iw = w;
                const int n_itr = P.angle_ticks;
                for (int s = 0; s < n_itr; s++) {
                    f3 wv = iw;
                    float ts = dt / n_itr;
                    for (int k = 0; k < 2; k++) {
                        f3 Iw = mul(it, wv);
                        f3 f = ts * cross(wv, Iw) - mul(it, iw - wv);
                        M33 cw = mul(crossm(wv), it), ci = crossm(Iw);
                        M33 jac;
                        for (int m = 0; m < 9; m++) jac.m[m] = it.m[m] + ts * (cw.m[m] - ci.m[m]);
                        if (fabsf(det(jac)) > 0.00000000001f) wv = wv - mul(inverse(jac), f);
                    }
                    iw = wv;
                    iq = qmul(qaxis(ts * mag(iw), iw), iq);
                    if (s + 1 < n_itr) {
                        M33 R = quatRot(iq), Rc = quatRot(qconj(iq));
                        it = mul(mul(R, Iref), Rc);
                    }
                }
                q = iq;
                w = iw;
            }
            q = qmul(qaxis(dt * mag(pw), pw), q);
        }
        // RigidBody::updateInertiaTensor (RigidBody.cpp:270-279)
        q = qnormalize(q);
        if (mv == 0) {
            M33 R = quatRot(q), Rc = quatRot(qconj(q));
            store9(d.iw + 9 * i, mul(mul(R, load9(d.iref + 9 * i)), Rc));
            store9(d.iinv + 9 * i, mul(mul(R, load9(d.iinv_ref + 9 * i)), Rc));
        }
        if (!(isfinite(c.x) && isfinite(c.y) && isfinite(c.z) && isfinite(q.x))) atomicOr(d.status, ST_NAN);
        d.pos[i] = pos;
        d.rot[i] = q;
        d.angv[i] = make_float4(w.x, w.y, w.z, 0.f);
        d.pvel[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        d.pangv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (last) {
            bool moved = pos.x != pos0.x || pos.y != pos0.y || pos.z != pos0.z || q.x != q0.x || q.y != q0.y || q.z != q0.z || q.w != q0.w;
            d.moved[i] = moved;
        }
    }
}

// External state write (cpgpu_batch_write_state): velocities are taken as
// given; a body whose pose changed gets its world inertia tensors and AABB
// recomputed from the new pose, an unchanged body keeps them bit for bit.
__global__ void k_apply_state(Dev d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_bodies; i += gridDim.x * blockDim.x) {
        const float4 p = d.stage[4 * i], q = d.stage[4 * i + 1], v = d.stage[4 * i + 2], w = d.stage[4 * i + 3];
        if (d.movement[i] != 1) {
            d.vel[i] = make_float4(v.x, v.y, v.z, 0.f);
            d.angv[i] = make_float4(w.x, w.y, w.z, 0.f);
        }
        const float4 p0 = d.pos[i], q0 = d.rot[i];
        if (p.x == p0.x && p.y == p0.y && p.z == p0.z && q.x == q0.x && q.y == q0.y && q.z == q0.z && q.w == q0.w) continue;
        d.pos[i] = make_float4(p.x, p.y, p.z, p0.w);
        d.rot[i] = q;
        M33 R = quatRot(q), Rc = quatRot(qconj(q));
        if (d.movement[i] == 0) {
            store9(d.iw + 9 * i, mul(mul(R, load9(d.iref + 9 * i)), Rc));
            store9(d.iinv + 9 * i, mul(mul(R, load9(d.iinv_ref + 9 * i)), Rc));
        }
        f3 mn, mx;
        shape_aabb(d.shapes + d.shape[i], mk(p), R, &mn, &mx);
        d.aabb_lo[i] = make_float4(mn.x, mn.y, mn.z, 0.f);
        d.aabb_hi[i] = make_float4(mx.x, mx.y, mx.z, 0.f);
    }
}

// host-layout state rows (pos, rot, vel, ang vel per body) of a batch split
// into parts: each part gathers / scatters its bodies' rows by index
__global__ void k_gather_state(const float4* __restrict__ all, const int* __restrict__ rows, int n, float4* __restrict__ stage) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int r = rows[i];
        for (int k = 0; k < 4; k++) stage[4 * i + k] = all[4 * (size_t)r + k];
    }
}
__global__ void k_scatter_state(Dev d, const int* __restrict__ rows, float4* __restrict__ all) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_bodies; i += gridDim.x * blockDim.x) {
        float4* o = all + 4 * (size_t)rows[i];
        o[0] = d.pos[i]; o[1] = d.rot[i]; o[2] = d.vel[i]; o[3] = d.angv[i];
    }
}

int grid_for(int n, int per_block, int n_sms) {
    int g = (n + per_block - 1) / per_block;
    int cap = n_sms * 8;
    return g < 1 ? 1 : (g > cap ? cap : g);
}

}  // namespace

void launch_rows(const Dev& d, int first, int last, const Launch& L) {
    k_rows<<<L.n_sms * 8, 128, 0, L.st>>>(d, first, last);
}

int pgs_big_smem_bytes(int dv_cap) {
    return 64 + kRingSlots * kChunkRows * (int)sizeof(RowBlock) + (dv_cap + 1) * 16 * kDvF4;
}

// blocks of k_pgs_big resident per SM for this Δv capacity (one chain each)
int pgs_big_blocks_per_sm(int dv_cap) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_pgs_big<true>, 32, pgs_big_smem_bytes(dv_cap)) != cudaSuccess || n < 1) n = 1;
    return n;
}

// The attribute is the kernel's, shared by every batch of the process: it is
// set for the largest Δv area any batch uses, so that a batch built later with
// a smaller one does not lower the limit under an earlier batch's launches
void prepare_pgs(int dv_cap) {
    (void)dv_cap;
    cudaFuncSetAttribute(k_pgs_joint, cudaFuncAttributeMaxDynamicSharedMemorySize, kJointSmem);
    cudaFuncSetAttribute(k_pgs_big<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, pgs_big_smem_bytes(kPgsDvCapMax));
}

void launch_pgs_schedule(const Dev& d, const Launch& L) {
    k_sched_count<<<L.n_sms * 2, 256, 0, L.st>>>(d);
    k_sched_place<<<L.n_sms * 2, 256, 0, L.st>>>(d);
}

void launch_pgs_joint(const Dev& d, bool first, int dv_cap, const Launch& L) {
    if (d.n_joint_edges == 0) return;
    k_pgs_joint<<<L.n_sms * 3, 32, kJointSmem, L.st>>>(d, first ? 1 : 0, std::min(dv_cap, kJointDv));
}

void launch_pgs(const Dev& d, int dv_cap, int max_world, int big_blocks, const Branches& b, const Launch& L) {
    // large islands on the main stream, middling and small ones (and islands
    // whose Δv does not fit in shared memory, where a world is large enough to
    // hold one) concurrently on side branches
    cudaMemsetAsync(d.sched + kBigNext, 0, 4 * sizeof(int), L.st);
    cudaEventRecord(b.fork, L.st);
    cudaStreamWaitEvent(b.side, b.fork, 0);
    cudaStreamWaitEvent(b.side2, b.fork, 0);
    if (max_world > dv_cap) k_pgs_big<false><<<L.n_sms, 32, pgs_big_smem_bytes(0), b.side>>>(d, dv_cap);
    k_pgs_small<<<L.n_sms * 8, 64, 0, b.side>>>(d);
    cudaEventRecord(b.join, b.side);
    k_pgs_mid<<<L.n_sms * 10, 32, kMidSmem, b.side2>>>(d, L.n_sms * 2);
    cudaEventRecord(b.join2, b.side2);
    k_pgs_big<true><<<big_blocks, 32, pgs_big_smem_bytes(dv_cap), L.st>>>(d, dv_cap);
    cudaStreamWaitEvent(L.st, b.join, 0);
    cudaStreamWaitEvent(L.st, b.join2, 0);
}

void launch_integrate(const Dev& d, int last, const Launch& L) {
    k_integrate<<<grid_for(d.n_bodies, 128, L.n_sms), 128, 0, L.st>>>(d, last);
}

void launch_apply_state(const Dev& d, const Launch& L) {
    k_apply_state<<<grid_for(d.n_bodies, 128, L.n_sms), 128, 0, L.st>>>(d);
}

void launch_gather_state(const Dev& d, const float4* all, const int* rows, const Launch& L) {
    k_gather_state<<<grid_for(d.n_bodies, 128, L.n_sms), 128, 0, L.st>>>(all, rows, d.n_bodies, d.stage);
}

void launch_scatter_state(const Dev& d, const int* rows, float4* all, const Launch& L) {
    k_scatter_state<<<grid_for(d.n_bodies, 128, L.n_sms), 128, 0, L.st>>>(d, rows, all);
}

}  // namespace cpgpu
