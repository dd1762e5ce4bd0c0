// XPBD constraint solves, integration and velocity passes on the device.
//
// Two lanes of a warp solve one solver node (a broad-phase pair with its contacts, or one external
// joint) in FP32, one lane per body (Duo; the FP64 solves are in rp_exact.cuh): each lane loads its body into
// registers, applies the corrections in the reference's order and writes it back once; nodes of one level
// never share a non-fixed body, so no two lanes write the same body. The corrections of the two bodies differ
// only in sign, so the second body's lane works on negated vectors (separation, normal, impulse): negation is
// exact, every product and sum rounds as in the one-thread form, and both lanes take the same branches.
// What bounds a node is the instruction stream of one warp with two active lanes: a contact is
// about a thousand dependent instructions in the one-thread form. Half of them belong to each body,
// so the lane pair halves the stream.
//
// EXACT=true mirrors the reference's FP64 expressions term for term (built without FMA
// contraction it reproduces the reference bit for bit). EXACT=false keeps positions and
// orientations in FP64 and does the rest in FP32, forming position differences in FP64 before
// rounding so that precision does not depend on the distance from the world origin.
//
// References (raw-physics): pbd.cpp:81-406 (solves), :537-577 (predict), :623-643 (velocity
// update), :646-740 (velocity solver); pbd_base_constraints.cpp:6-227; physics_util.cpp:5-63.
#pragma once
#include "rp_math.cuh"
#include "rp_world.h"

namespace rp {

constexpr double PI_REF = 3.14159265358979;   // PI_F of include/gm.h:8

// Rotation used for the working-precision algebra of a body.
template <typename R>
__device__ __forceinline__ Qt<R> wq(const Qt<double>& q) { return qcast<R>(q); }

// --------------------------------------------------------------------------------------------
// The lane pair of one solver node: lanes 2i and 2i + 1 of a warp hold the node's first and second
// body. Both lanes of a pair always call these together.
struct Duo {
    unsigned mask;
    int side;          // 0: the node's first body, 1: its second
    bool second_right; // FP32 contacts: this lane's sums are fused as a second body's (see JOINT)
    template <typename T> __device__ __forceinline__ T other(T v) const { return __shfl_xor_sync(mask, v, 1); }
    template <typename T> __device__ __forceinline__ V3<T> other(V3<T> v) const { return v3<T>(other(v.x), other(v.y), other(v.z)); }
    template <typename T> __device__ __forceinline__ Qt<T> other(Qt<T> q) const {
        return qt<T>(other(q.x), other(q.y), other(q.z), other(q.w));
    }
    // the vector as the first body sees it, from this lane's body's side
    template <typename T> __device__ __forceinline__ V3<T> own(V3<T> v) const {
        return side ? v3<T>(-v.x, -v.y, -v.z) : v;
    }
    // the first / second body's value, given this lane's value and the other's
    template <typename V> __device__ __forceinline__ V first(const V& mine, const V& theirs) const { return side ? theirs : mine; }
    template <typename V> __device__ __forceinline__ V second(const V& mine, const V& theirs) const { return side ? mine : theirs; }
};

__device__ __forceinline__ Duo duo_of_lane() {
    const unsigned lane = threadIdx.x & 31u;
    return Duo{3u << (lane & 30u), (int)(lane & 1u), (lane & 1u) != 0u};
}

// Normalisation of an FP64 quaternion in the FP32 build: an FP32 reciprocal square root refined by
// one FP64 Newton step (relative error ~1e-14), instead of an FP64 square root and four FP64
// divisions, which GB300 executes at a small fraction of its FP32 rate.
__device__ __forceinline__ Qt<double> qnormalize_fast(Qt<double> q) {
    // (roundings spelled out: every kernel that normalises gives the same bits)
    const double n2 = __fma_rn(q.w, q.w, __fma_rn(q.z, q.z, __fma_rn(q.x, q.x, __dmul_rn(q.y, q.y))));
    double r = (double)rsqrtf((float)n2);
    r = __dmul_rn(r, __fma_rn(-__dmul_rn(__dmul_rn(0.5, n2), r), r, 1.5));
    return qt<double>(q.x * r, q.y * r, q.z * r, q.w * r);
}

// limit_angle (pbd.cpp:175-217)
// Joint limits are evaluated in FP64 in both builds (the axes come from the FP64 orientations):
// asin's slope diverges at |s| -> 1, so at a +-90 degree limit an FP32 s (error 1e-7) would move
// phi by sqrt(2e-7) ~ 4.5e-4 rad; in FP64 the same amplification stays below 1e-7.
template <typename R>
__device__ bool limit_angle(V3<R> n, V3<R> n1, V3<R> n2, R alpha, R beta, V3<R>& dq) {
    const R pi = (R)PI_REF;
    R phi = asin(vdot(vcross(n1, n2), n));
    if (vdot(n1, n2) < (R)0) phi = pi - phi;
    if (phi > pi) phi = phi - (R)2.0 * pi;
    if (phi < -pi) phi = phi + (R)2.0 * pi;
    if (phi < alpha || phi > beta) {
        phi = (phi > beta) ? beta : ((phi < alpha) ? alpha : phi);
        V3<R> ax = n;
        if (vlen(ax) != (R)0) ax = vnorm(ax);
        R s = sin(phi / (R)2.0);
        Qt<R> rot = qt<R>(ax.x * s, ax.y * s, ax.z * s, cos(phi / (R)2.0));
        n1 = qrotate(rot, n1);
        dq = vcross(n1, n2);
        return true;
    }
    return false;
}

// True when limit_angle could apply a correction. With limits at or beyond +-pi the wrapped angle
// can never leave them (any build). Otherwise, in the FP32 build, an FP32 estimate of the angle from
// FP32 axes decides when it lies more than 0.01 rad inside both limits: its error stays below 1e-3 rad
// even where asin is ill-conditioned (|s| -> 1). Near a limit, near the +-pi wrap, or where the
// branch on <n1, n2> is within 1e-3 of flipping, the FP64 evaluation runs.
__device__ __forceinline__ bool limit_may_act(V3<float> n, V3<float> n1, V3<float> n2, double lo, double hi) {
    if (lo <= -PI_REF && hi >= PI_REF) return false;
    if (lo < -PI_REF + 0.02 || hi > PI_REF - 0.02) return true;
    const float c = vdot(n1, n2);
    if (fabsf(c) < 1e-3f) return true;
    const float pi = (float)PI_REF;
    float phi = asinf(fminf(fmaxf(vdot(vcross(n1, n2), n), -1.f), 1.f));
    if (c < 0.f) phi = pi - phi;
    if (phi > pi) phi -= 2.f * pi;
    if (phi < -pi) phi += 2.f * pi;
    return !(phi >= (float)lo + 0.01f && phi <= (float)hi - 0.01f);
}

// --------------------------------------------------------------------------------------------
// FP32 build: a node's bodies as an FP64 base pose plus FP32 deltas.
//
// A solver node applies a handful of small corrections to its two bodies. Each body's pose is read
// once in FP64 (x0, q0); corrections accumulate in FP32 deltas (dx, dq) relative to it, and the FP64
// pose is written back once: x = x0 + dx, q = normalize(q0 + dq). The renormalisation after every
// orientation update (pbd_base_constraints.cpp:83-103) is carried out exactly in delta form:
// with u = dq + increment and e = |q0 + u|^2 - 1 = 2 q0.u + u.u, the normalised quaternion is
// q0 + q0 (r - 1) + u r with r - 1 = -e / (s (1 + s)), s = sqrt(1 + e), all of which are small,
// well-conditioned FP32 quantities. Per contact the solve then needs no FP64 arithmetic at all.
// FP32 build: a body during the substep's position sweep. Its FP64 pose stays at the predicted pose
// (pos / rot); the sweep's corrections accumulate per body in FP32 deltas (sdx, sdq), and the pose is
// folded into FP64 once per substep (fold_body), so FP64 carries the pose across substeps while the
// solve itself runs in FP32. A node loads the body's FP32 orientation (pose_f) and deltas and stores
// the deltas back.
struct FBody {
    V3<float> dx;
    Qt<float> q0f, dq;
    float invm;
    float S[6];   // local inverse inertia, symmetric storage (xx yy zz xy xz yz)
    bool fixed;
    int idx;
    __device__ __forceinline__ Qt<float> q() const {
        return qt<float>(__fadd_rn(q0f.x, dq.x), __fadd_rn(q0f.y, dq.y), __fadd_rn(q0f.z, dq.z), __fadd_rn(q0f.w, dq.w));
    }
};

__device__ __forceinline__ FBody load_fbody(const WorldView<float>& W, int b) {
    FBody B;
    const float4 qf = W.pose_f[2 * b + 1], d = W.sdx[b], q = W.sdq[b];
    B.q0f = qt<float>(qf.x, qf.y, qf.z, qf.w);
    B.dx = v3<float>(d.x, d.y, d.z);
    B.dq = qt<float>(q.x, q.y, q.z, q.w);
    B.invm = W.inv_mass[b];
#pragma unroll
    for (int i = 0; i < 6; ++i) B.S[i] = W.inv_inertia[6 * b + i];
    B.fixed = W.fixed[b] != 0;
    B.idx = b;
    return B;
}

__device__ __forceinline__ void store_fbody(const WorldView<float>& W, const FBody& B) {
    if (B.fixed) return;
    W.sdx[B.idx] = make_float4(B.dx.x, B.dx.y, B.dx.z, 0.f);
    W.sdq[B.idx] = make_float4(B.dq.x, B.dq.y, B.dq.z, B.dq.w);
}

// (float)(x_a - x_b) of two bodies' predicted positions, as stored in pair_base
__device__ __forceinline__ float4 fbase4(const WorldView<float>& W, int a, int b) {
    const double4_32a pa = W.pos[a], pb = W.pos[b];
    return make_float4((float)(pa.x - pb.x), (float)(pa.y - pb.y), (float)(pa.z - pb.z), 0.f);
}


// The position sweep's corrections d, q into the FP64 pose (x += dx, q = normalize(q + dq)); false for a body
// the sweep did not touch, which keeps its pose.
__device__ __forceinline__ bool fold_pose(double4_32a& p4, double4_32a& q4, float4 d, float4 q) {
    if (d.x == 0.f && d.y == 0.f && d.z == 0.f && q.x == 0.f && q.y == 0.f && q.z == 0.f && q.w == 0.f) return false;
    const Qt<double> nq = qnormalize_fast(qt<double>(q4.x + (double)q.x, q4.y + (double)q.y, q4.z + (double)q.z,
                                                     q4.w + (double)q.w));
    p4 = make_double4_32a(p4.x + (double)d.x, p4.y + (double)d.y, p4.z + (double)d.z, 0.0);
    q4 = make_double4_32a(nq.x, nq.y, nq.z, nq.w);
    return true;
}
// for one body in global memory, with the FP32 orientation copy the velocity sweep reads
__device__ __forceinline__ void fold_body(const WorldView<float>& W, int b) {
    double4_32a p = W.pos[b], q = W.rot[b];
    if (!fold_pose(p, q, W.sdx[b], W.sdq[b])) return;
    W.pos[b] = p;
    W.rot[b] = q;
    W.pose_f[2 * b + 1] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
}

// JOINT in the functions below: the contact solve and the joint solves fuse some of their sums in
// different order (the last step of frot_update, the y component of R^T v; the xy elements of a
// contact's second body, D.second_right), and each keeps its own.

// q <- normalize(q + inc), in delta form
template <bool JOINT>
__device__ __forceinline__ void frot_update(FBody& B, Qt<float> inc) {
    const Qt<float> u = qt<float>(__fadd_rn(B.dq.x, inc.x), __fadd_rn(B.dq.y, inc.y), __fadd_rn(B.dq.z, inc.z), __fadd_rn(B.dq.w, inc.w));
    const float d = __fmaf_rn(B.q0f.w, u.w, sum3(B.q0f.x, u.x, B.q0f.y, u.y, B.q0f.z, u.z));
    const float e = __fmaf_rn(2.f, d, __fmaf_rn(u.w, u.w, sum3(u.x, u.x, u.y, u.y, u.z, u.z)));
    const float u1 = __fadd_rn(1.f, e);   // |q0 + u|^2, close to 1
    const float s = __fmul_rn(u1, rsqrtf(u1));
    const float rm1 = __fdividef(-e, __fmul_rn(s, __fadd_rn(1.f, s)));
    const float r = __fadd_rn(1.f, rm1);
    if (JOINT)
        B.dq = qt<float>(sum2(B.q0f.x, rm1, u.x, r), sum2(u.y, r, B.q0f.y, rm1), sum2(u.z, r, B.q0f.z, rm1), sum2(u.w, r, B.q0f.w, rm1));
    else
        B.dq = qt<float>(sum2(B.q0f.x, rm1, u.x, r), sum2(B.q0f.y, rm1, u.y, r), sum2(B.q0f.z, rm1, u.z, r), sum2(B.q0f.w, rm1, u.w, r));
}

// FP32 delta-form arithmetic: unit vectors from the reciprocal square root of the special-function
// unit and divisions by __fdividef (each within 2 ulp), shorter dependent chains than IEEE sqrtf and
// division in the serial Gauss-Seidel chains; squared lengths at or below 1e-36 take the IEEE path
// (rsqrtf flushes subnormal inputs).
__device__ __forceinline__ float funit(V3<float> v, V3<float>& n) {
    const float c2 = dot_f(v, v);
    if (c2 > 1e-36f) {
        const float r = rsqrtf(c2);
        n = scale_f(r, v);
        return __fmul_rn(c2, r);
    }
    const float c = sqrtf(c2);
    if (c > 0.f) n = v3<float>(v.x / c, v.y / c, v.z / c);
    return c;
}

// The world inverse inertia applied to v at the body's current orientation, R (S (R^T v)): the
// products the reference forms with the world tensor R S R^T (physics_util.cpp:26-63), without
// keeping the tensor itself live through the solve (the FP32 path's register budget).
template <bool JOINT>
__device__ __forceinline__ V3<float> fIinv(const Duo& D, const FBody& B, V3<float> v) {
    const M3<float> R = mat3_f(B.q(), !JOINT && D.second_right);
    const V3<float> l = v3<float>(sum3(R.d[0][0], v.x, R.d[1][0], v.y, R.d[2][0], v.z),
                                  JOINT ? sum3(R.d[1][1], v.y, R.d[0][1], v.x, R.d[2][1], v.z)
                                        : sum3(R.d[0][1], v.x, R.d[1][1], v.y, R.d[2][1], v.z),
                                  sum3(R.d[0][2], v.x, R.d[1][2], v.y, R.d[2][2], v.z));
    const V3<float> t = v3<float>(sum3(B.S[0], l.x, B.S[3], l.y, B.S[4], l.z), sum3(B.S[3], l.x, B.S[1], l.y, B.S[5], l.z),
                                  sum3(B.S[4], l.x, B.S[5], l.y, B.S[2], l.z));
    return mulv_f(R, t);
}

// the generalised inverse mass of this lane's body for a correction along unit n at anchor r
template <bool JOINT>
__device__ __forceinline__ float fmass(const Duo& D, const FBody& B, V3<float> r, V3<float> n) {
    const V3<float> c = cross_f(r, n);
    return __fadd_rn(B.invm, dot_f(c, fIinv<JOINT>(D, B, c)));
}

// the angular part of a correction: q <- normalize(q + (a, 0) q / 2)
template <bool JOINT>
__device__ __forceinline__ void fturn(FBody& B, V3<float> a) {
    const Qt<float> q = qmul_pure_f(a, B.q());
    if (!B.fixed) frot_update<JOINT>(B, qt<float>(0.5f * q.x, 0.5f * q.y, 0.5f * q.z, 0.5f * q.w));
}

__device__ __forceinline__ float fpos_dlambda(const Duo& D, const FBody& B, V3<float> r, V3<float> dx) {
    V3<float> n;
    const float c = funit(dx, n);
    if (c <= 0.f) return 0.f;
    const float w = fmass<false>(D, B, r, n);
    return __fdividef(-c, __fadd_rn(w, D.other(w)));   // contacts carry zero compliance (pbd.cpp:123,133)
}

template <bool JOINT>
__device__ __forceinline__ void fpos_apply(const Duo& D, FBody& B, V3<float> r, float dl, V3<float> dx) {
    V3<float> n;
    const float c = funit(dx, n);
    if (c <= 0.f) return;
    const V3<float> imp = scale_f(dl, n);
    if (!B.fixed) B.dx = axpy_f(B.invm, imp, B.dx);
    fturn<JOINT>(B, fIinv<JOINT>(D, B, cross_f(r, imp)));
}

// collision_constraint_solve (pbd.cpp:107-154) on FP32 deltas. rl: this body's anchor and multiplier
// (the first body's lane holds lambda_n, the second's lambda_t); n and base (the predicted positions'
// difference) seen from this body; pred_d, prev_qf: the substep's displacement and previous orientation by
// B.idx; returns this lane's multiplier.
static __device__ float fcollision_solve(const float4* pred_d, const float4* prev_qf, const Duo& D, FBody& B, V3<float> base, float4 rl, V3<float> n,
                                         float mus) {
    const V3<float> r_lc = v3<float>(rl.x, rl.y, rl.z);
    V3<float> r = rotate_f(B.q(), r_lc, true);
    const V3<float> gap = add_f(add_f(base, sub_f(B.dx, D.other(B.dx))), sub_f(r, D.other(r)));
    const float d = sum3(gap.y, n.y, gap.x, n.x, gap.z, n.z);
    if (!(d > 0.f)) return rl.w;
    const float lo = D.other(rl.w);
    float lambda_n = D.first(rl.w, lo), lambda_t = D.second(rl.w, lo);
    const V3<float> dx = scale_f(d, n);
    float dl = fpos_dlambda(D, B, r, dx);
    fpos_apply<false>(D, B, r, dl, dx);
    lambda_n = __fadd_rn(lambda_n, dl);
    r = rotate_f(B.q(), r_lc, D.second_right, D.second_right);
    dl = fpos_dlambda(D, B, r, dx);
    const float lt = __fadd_rn(lambda_t, dl);
    if (lt > __fmul_rn(mus, lambda_n)) {
        // displacement since the substep began: the predict step's (pred_d, FP32 from the FP64 poses)
        // plus the sweep's; the previous orientation's FP32 copy (prev_qf)
        const float4 pd = pred_d[B.idx], qp = prev_qf[B.idx];
        const V3<float> u = add_f(add_f(v3<float>(pd.x, pd.y, pd.z), B.dx),
                                  sub_f(r, rotate_f(qt<float>(qp.x, qp.y, qp.z, qp.w), r_lc)));
        const V3<float> dp = sub_f(u, D.other(u));
        fpos_apply<false>(D, B, r, dl, axpy_f(-dot_f(dp, n), n, dp));
        lambda_t = lt;
    }
    return D.side ? lambda_t : lambda_n;
}

// --------------------------------------------------------------------------------------------
// External constraints of the FP32 build on FP64-base / FP32-delta bodies (pbd.cpp:81-379): the
// same order of corrections as ext_solve, each applied to the FP32 deltas; joint-limit angles are
// screened in FP32 and evaluated in FP64 (from the FP64 orientation q0 + dq) where they may act.
__device__ __forceinline__ float fdlambda(float c, float w1, float w2, float h, float compliance, float lambda) {
    const float til = __fdividef(compliance, __fmul_rn(h, h));
    return __fdividef(__fmaf_rn(-til, lambda, -c), __fadd_rn(__fadd_rn(w1, w2), til));
}

__device__ __forceinline__ float fpos_dlambda_c(const Duo& D, const FBody& B, V3<float> r, float h, float compliance, float lambda,
                                                V3<float> dx) {
    V3<float> n;
    const float c = funit(dx, n);
    if (c <= 0.f) return 0.f;
    const float w = fmass<true>(D, B, r, n);
    return fdlambda(c, w, D.other(w), h, compliance, lambda);
}

// angular corrections of this lane's body (pbd_base_constraints.cpp:125-227)
__device__ __forceinline__ float fang_dlambda(const Duo& D, const FBody& B, float h, float compliance, float lambda, V3<float> dq) {
    V3<float> n;
    const float th = funit(dq, n);
    if (th <= 0.f) return 0.f;
    const float w = dot_f(n, fIinv<true>(D, B, n));
    return fdlambda(th, w, D.other(w), h, compliance, lambda);
}

__device__ __forceinline__ void fang_apply(const Duo& D, FBody& B, float dl, V3<float> dq) {
    V3<float> n;
    const float th = funit(dq, n);
    if (th <= 0.f) return;
    fturn<true>(B, fIinv<true>(D, B, scale_f(-dl, n)));
}

// What the FP32 solve of one joint reads of it, besides its bodies: the axes and limits, this lane's body's
// anchor, and the difference of the predicted positions (minus the rest offset of a positional joint).
struct JointF {
    int type, a1, a2, l1, l2;
    bool limited;
    float compliance;
    V3<float> r1, r2, base;
    double lo, hi, lo2, hi2;
};

// A joint as the solve kernels stage it: the FP32 operands rounded at upload, and the position difference
// formed in FP64 and rounded once per substep (the poses do not change during the position sweep).
__device__ __forceinline__ JointF load_joint(const WorldView<float>& W, const ExtConstraint& C) {
    JointF j;
    j.type = C.type;
    j.a1 = C.a1; j.a2 = C.a2; j.l1 = C.l1; j.l2 = C.l2;
    j.limited = C.limited != 0;
    j.compliance = C.compliance_f;
    j.r1 = v3<float>(C.r1f[0], C.r1f[1], C.r1f[2]);
    j.r2 = v3<float>(C.r2f[0], C.r2f[1], C.r2f[2]);
    j.lo = C.lo; j.hi = C.hi; j.lo2 = C.lo2; j.hi2 = C.hi2;
    const double4_32a pa = W.pos[C.e1], pb = W.pos[C.e2];
    double x = pa.x - pb.x, y = pa.y - pb.y, z = pa.z - pb.z;
    if (C.type == CON_POSITIONAL) { x -= C.distance[0]; y -= C.distance[1]; z -= C.distance[2]; }
    j.base = v3<float>((float)x, (float)y, (float)z);
    return j;
}

// FP64 evaluation of a joint limit that the FP32 screen could not rule out (rare): kind 0 the hinge
// limit (pbd.cpp:279-298), 1 the spherical swing limit, 2 the spherical twist limit (pbd.cpp:327-378),
// from the FP64 orientations q0 + dq of the first and the second body; true with the correction dq as
// the first body sees it. Out of line, so that the joint solve's common path keeps its values in
// registers; both lanes of a pair evaluate it on the same values.
static __device__ __noinline__ bool flimit64(Qt<double> qa, Qt<double> qb, const JointF& C, int kind, V3<float>& dq) {
    const double EPS64 = 1e-50;
    V3<double> dq64;
    bool act = false;
    if (kind == 0) {
        act = limit_angle<double>(qaxis(qa, C.a1), qaxis(qa, C.l1), qaxis(qb, C.l2), C.lo, C.hi, dq64);
    } else if (kind == 1) {
        const V3<double> n1 = qaxis(qa, C.a1), n2 = qaxis(qb, C.a2);
        const V3<double> n = vcross(n1, n2);
        const double nl = vlen(n);
        act = nl > EPS64 && limit_angle<double>(v3<double>(n.x / nl, n.y / nl, n.z / nl), n1, n2, C.lo, C.hi, dq64);
    } else {
        const V3<double> a1 = qaxis(qa, C.a1), b1 = qaxis(qa, C.l1), a2 = qaxis(qb, C.a2), b2 = qaxis(qb, C.l2);
        V3<double> n = vadd(a1, a2);
        const double nl = vlen(n);
        if (nl > EPS64) {
            n = v3<double>(n.x / nl, n.y / nl, n.z / nl);
            const V3<double> n1 = vsub(b1, vscale(vdot(n, b1), n)), n2 = vsub(b2, vscale(vdot(n, b2), n));
            const double l1 = vlen(n1), l2 = vlen(n2);
            act = l1 > EPS64 && l2 > EPS64 &&
                  limit_angle<double>(n, v3<double>(n1.x / l1, n1.y / l1, n1.z / l1), v3<double>(n2.x / l2, n2.y / l2, n2.z / l2),
                                      C.lo2, C.hi2, dq64);
        }
    }
    if (act) dq = v3cast<float>(dq64);
    return act;
}

// an axis of a body in world coordinates, FP32 with its roundings spelled out (qaxis)
__device__ __forceinline__ V3<float> axis_f(Qt<float> q, int axis) {
    const float x2 = 2.f * q.x, y2 = 2.f * q.y, z2 = 2.f * q.z, w = axis & 1 ? q.w : -q.w, w2 = 2.f * w;
    if (axis < 2) return v3<float>(__fmaf_rn(-z2, q.z, __fmaf_rn(-y2, q.y, 1.f)), dif2(x2, q.y, w2, q.z), sum2(x2, q.z, w2, q.y));
    if (axis < 4) return v3<float>(sum2(x2, q.y, w2, q.z), __fmaf_rn(-z2, q.z, __fmaf_rn(-x2, q.x, 1.f)), dif2(y2, q.z, w2, q.x));
    return v3<float>(dif2(x2, q.z, w2, q.y), sum2(y2, q.z, w2, q.x), __fmaf_rn(-y2, q.y, __fmaf_rn(-x2, q.x, 1.f)));
}

// One joint on this lane's body B. rot: the body's predicted FP64 orientation (read only where a limit
// has to be decided in FP64). lam: the joint's Lagrange multipliers of the substep as FP32 (they start at
// zero every substep and enter only through compliance): zero in its first sweep; both lanes hold them.
static __device__ void fext_solve(const Duo& D, FBody& B, const double4_32a* rot, const JointF& C, float (&lam)[3], float h) {
    const V3<float> r_lc = D.side ? C.r2 : C.r1;
    const V3<float> base = D.own(C.base);
    // one positional correction along dx at anchor r
    auto positional = [&](float compliance, V3<float> r, V3<float> dx) {
        const float dl = fpos_dlambda_c(D, B, r, h, compliance, lam[0], dx);
        fpos_apply<true>(D, B, r, dl, dx);
        lam[0] = __fadd_rn(lam[0], dl);
    };
    auto angular = [&](float& l, float compliance, V3<float> dq) {
        const float dl = fang_dlambda(D, B, h, compliance, l, dq);
        fang_apply(D, B, dl, dq);
        l = __fadd_rn(l, dl);
    };
    // the anchors coincide (pbd.cpp:265-276, 303-314)
    auto attach = [&]() {
        const V3<float> r = rotate_f(B.q(), r_lc);
        positional(0.f, r, add_f(add_f(base, sub_f(B.dx, D.other(B.dx))), sub_f(r, D.other(r))));
    };
    // an axis of the first and of the second body, in both lanes
    auto axes = [&](int k1, int k2, V3<float>& u1, V3<float>& u2) {
        const V3<float> mine = axis_f(B.q(), D.side ? k2 : k1), theirs = D.other(mine);
        u1 = D.first(mine, theirs);
        u2 = D.second(mine, theirs);
    };
    // a limit the FP32 screen could not rule out
    auto limit = [&](int kind) {
        const double4_32a q4 = *rot;
        const Qt<double> q = qt<double>(q4.x + (double)B.dq.x, q4.y + (double)B.dq.y, q4.z + (double)B.dq.z, q4.w + (double)B.dq.w);
        const Qt<double> o = D.other(q);
        V3<float> dq;
        const JointF c = C;   // a copy: the call takes an address, which would keep the joint in local memory
        if (flimit64(D.first(q, o), D.second(q, o), c, kind, dq)) angular(kind == 1 ? lam[1] : lam[2], 0.f, D.own(dq));
    };
    switch (C.type) {
    case CON_POSITIONAL:   // pbd.cpp:81-97
        positional(C.compliance, rotate_f(B.q(), r_lc), add_f(base, sub_f(B.dx, D.other(B.dx))));
        break;
    case CON_MUTUAL_ORIENTATION: {  // pbd.cpp:156-173
        const Qt<float> mq = B.q(), oq = D.other(mq);
        const Qt<float> aux = qmul(D.first(mq, oq), qinverse(D.second(mq, oq)));
        angular(lam[0], C.compliance, D.own(v3<float>(2.f * aux.x, 2.f * aux.y, 2.f * aux.z)));
    } break;
    case CON_HINGE: {  // pbd.cpp:245-299
        V3<float> u1, u2;
        axes(C.a1, C.a2, u1, u2);
        angular(lam[1], C.compliance, D.own(cross_f(u1, u2)));
        attach();
        if (C.limited) {
            V3<float> n1, n2;
            axes(C.a1, C.a2, u1, u2);
            axes(C.l1, C.l2, n1, n2);
            if (limit_may_act(u1, n1, n2, C.lo, C.hi)) limit(0);
        }
    } break;
    case CON_SPHERICAL: {  // pbd.cpp:301-379
        attach();
        if (!(C.lo <= -PI_REF && C.hi >= PI_REF)) {   // swing; limits at or beyond +-pi never act
            V3<float> f1, f2;
            axes(C.a1, C.a2, f1, f2);
            const V3<float> fn = vcross(f1, f2);
            const float fl = vlen(fn);
            if (fl < 1e-3f || limit_may_act(vscale(1.f / fl, fn), f1, f2, C.lo, C.hi)) limit(1);
        }
        if (!(C.lo2 <= -PI_REF && C.hi2 >= PI_REF)) {   // twist, on the orientations after the swing correction
            V3<float> f1, f2, g1, g2;
            axes(C.a1, C.a2, f1, f2);
            axes(C.l1, C.l2, g1, g2);
            V3<float> gn = vadd(f1, f2);
            const float gl = vlen(gn);
            bool act = true;
            if (gl >= 1e-3f) {
                gn = vscale(1.f / gl, gn);
                const V3<float> h1 = vsub(g1, vscale(vdot(gn, g1), gn)), h2 = vsub(g2, vscale(vdot(gn, g2), gn));
                const float l1 = vlen(h1), l2 = vlen(h2);
                act = l1 < 1e-3f || l2 < 1e-3f || limit_may_act(gn, vscale(1.f / l1, h1), vscale(1.f / l2, h2), C.lo2, C.hi2);
            }
            if (act) limit(2);
        }
    } break;
    default: break;
    }
}

// Predict (pbd.cpp:537-577): the pose x, q and velocities v, w of an awake body after a step h under force F and
// torque T.
template <typename R, bool EXACT>
__device__ __forceinline__ void predict_values(V3<double>& x, Qt<double>& q, V3<R>& v, V3<R>& w, V3<R> F, V3<R> T, R invm,
                                               const R (&si)[6], const R (&sI)[6], double h) {
    R hR = (R)h;
    v = vadd(v, vscale(hR * invm, F));
    if (EXACT) x = vadd(x, v3cast<double>(vscale(hR, v)));
    else x = vadd(x, vscale(h, v3cast<double>(v)));
    Qt<R> qw = wq<R>(q);
    M3<R> Iinv = world_tensor(qw, msym(si)), I = world_tensor(qw, msym(sI));
    w = vadd(w, vscale(hR, mmulv(Iinv, vsub(T, vcross(w, mmulv(I, w))))));
    Qt<R> qd = qmul(qt<R>(w.x, w.y, w.z, (R)0), qw);
    if (EXACT) {
        q.x = q.x + h * 0.5 * (double)qd.x; q.y = q.y + h * 0.5 * (double)qd.y;
        q.z = q.z + h * 0.5 * (double)qd.z; q.w = q.w + h * 0.5 * (double)qd.w;
        q = qnormalize(q);
    } else {
        R s = hR * (R)0.5;
        q.x = q.x + (double)(s * qd.x); q.y = q.y + (double)(s * qd.y);
        q.z = q.z + (double)(s * qd.z); q.w = q.w + (double)(s * qd.w);
        q = qnormalize_fast(q);
    }
}

// Predict for one body, and with STAGE the copies the substep's phases work from: the FP32 pose, and in the
// FP32 build the predict step's displacement, the previous orientation and, for the sweeps that keep them
// in global memory (DELTAS), zero sweep deltas. Every load is issued before the first use.
template <typename R, bool EXACT, bool STAGE, bool DELTAS>
__device__ __forceinline__ void predict_body(const WorldView<R>& W, int b, double h) {
    const double4_32a p = W.pos[b], q4 = W.rot[b];
    const bool moves = !W.fixed[b] && W.active[b];
    V3<R> v = v3<R>(W.vel[3 * b], W.vel[3 * b + 1], W.vel[3 * b + 2]);
    V3<R> w = v3<R>(W.omega[3 * b], W.omega[3 * b + 1], W.omega[3 * b + 2]);
    const V3<R> F = v3<R>((R)W.force[3 * b], (R)W.force[3 * b + 1], (R)W.force[3 * b + 2]);
    const V3<R> T = v3<R>((R)W.torque[3 * b], (R)W.torque[3 * b + 1], (R)W.torque[3 * b + 2]);
    const R invm = W.inv_mass[b];
    R si[6], sI[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) { si[i] = W.inv_inertia[6 * b + i]; sI[i] = W.inertia[6 * b + i]; }
    V3<double> x = v3<double>(p.x, p.y, p.z);
    Qt<double> q = qt<double>(q4.x, q4.y, q4.z, q4.w);
    W.prev_pos[b] = p;
    W.prev_rot[b] = q4;
    if (moves) {
        predict_values<R, EXACT>(x, q, v, w, F, T, invm, si, sI, h);
        W.pos[b] = make_double4_32a(x.x, x.y, x.z, 0.0);
        W.rot[b] = make_double4_32a(q.x, q.y, q.z, q.w);
        W.vel[3 * b] = v.x; W.vel[3 * b + 1] = v.y; W.vel[3 * b + 2] = v.z;
        W.omega[3 * b] = w.x; W.omega[3 * b + 1] = w.y; W.omega[3 * b + 2] = w.z;
    }
    if (!STAGE) return;
    W.pose_f[2 * b] = make_float4((float)x.x, (float)x.y, (float)x.z, 0.f);
    W.pose_f[2 * b + 1] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
    if constexpr (!EXACT) {
        if (DELTAS) {
            W.sdx[b] = make_float4(0.f, 0.f, 0.f, 0.f);
            W.sdq[b] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        W.pred_d[b] = make_float4((float)(x.x - p.x), (float)(x.y - p.y), (float)(x.z - p.z), 0.f);
        W.prev_qf[b] = make_float4((float)q4.x, (float)q4.y, (float)q4.z, (float)q4.w);
    }
}

// PBD velocity update (pbd.cpp:623-643): the velocities of a body that went from pose pp, pq4 to p, q4 in a
// substep; inv_h = 1 / h.
template <typename R, bool EXACT>
__device__ __forceinline__ void velocity_values(double4_32a p, double4_32a q4, double4_32a pp, double4_32a pq4, double inv_h, V3<R>& v,
                                                V3<R>& w) {
    V3<double> dx = vsub(v3<double>(p.x, p.y, p.z), v3<double>(pp.x, pp.y, pp.z));
    if constexpr (EXACT) {
        v = vscale(inv_h, dx);
        Qt<double> dq = qmul(qt<double>(q4.x, q4.y, q4.z, q4.w), qinverse(qt<double>(pq4.x, pq4.y, pq4.z, pq4.w)));
        const double two = 2.0 * inv_h;   // the reference's 2 / h: the same double
        w = (dq.w >= 0.0) ? vscale(two, v3<double>(dq.x, dq.y, dq.z)) : vscale(-two, v3<double>(dq.x, dq.y, dq.z));
    } else {
        // only the pose differences are formed in FP64. With q = q_prev + d,
        // q * q_prev^-1 = (0, 0, 0, |q_prev|^2) + d * q_prev^-1, so its vector part is d * q_prev^-1.
        const R ih = (R)inv_h;
        v = vscale(ih, v3cast<R>(dx));
        // (differences of rounded poses, not fused with the normalisation they come from)
        Qt<R> d = qt<R>((R)__dsub_rn(q4.x, pq4.x), (R)__dsub_rn(q4.y, pq4.y), (R)__dsub_rn(q4.z, pq4.z), (R)__dsub_rn(q4.w, pq4.w));
        Qt<R> qpi = qinverse(qt<R>((R)pq4.x, (R)pq4.y, (R)pq4.z, (R)pq4.w));
        Qt<R> dq = qmul(d, qpi);
        R sgn = ((R)1 + dq.w >= (R)0) ? (R)2 * ih : (R)-2 * ih;
        w = v3<R>(sgn * dq.x, sgn * dq.y, sgn * dq.z);
    }
}

// for one body, from global memory
template <typename R, bool EXACT>
__device__ void velocity_body(const WorldView<R>& W, int b, double h) {
    if (W.fixed[b] || !W.active[b]) return;
#pragma unroll
    for (int i = 0; i < 3; ++i) { W.prev_vel[3 * b + i] = W.vel[3 * b + i]; W.prev_omega[3 * b + i] = W.omega[3 * b + i]; }
    V3<R> v, w;
    velocity_values<R, EXACT>(W.pos[b], W.rot[b], W.prev_pos[b], W.prev_rot[b], 1.0 / h, v, w);
    W.vel[3 * b] = v.x; W.vel[3 * b + 1] = v.y; W.vel[3 * b + 2] = v.z;
    W.omega[3 * b] = w.x; W.omega[3 * b + 1] = w.y; W.omega[3 * b + 2] = w.z;
}

// world_tensor with its roundings spelled out
__device__ __forceinline__ M3<float> world_tensor_f(Qt<float> q, const float S[6]) {
    const M3<float> r = mat3_f(q);
    M3<float> x, o;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        x.d[i][0] = sum3(r.d[i][0], S[0], r.d[i][1], S[3], r.d[i][2], S[4]);
        x.d[i][1] = sum3(r.d[i][0], S[3], r.d[i][1], S[1], r.d[i][2], S[5]);
        x.d[i][2] = sum3(r.d[i][0], S[4], r.d[i][1], S[5], r.d[i][2], S[2]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) o.d[i][j] = sum3(x.d[i][0], r.d[j][0], x.d[i][1], r.d[j][1], x.d[i][2], r.d[j][2]);
    return o;
}

// Velocity solver for one contact (pbd.cpp:646-711) of this lane's body, its roundings spelled out: vel, om its
// velocities, pv, pw those before the velocity update, r its anchor in world orientation, I its world inverse
// inertia, n the normal seen from it.
__device__ __forceinline__ void fcontact_velocity(const Duo& D, V3<float> r, const M3<float>& I, V3<float> n, float invm, bool fixed,
                                                  float lambda_n, float h, float mud, float e, V3<float>& vel, V3<float>& om,
                                                  V3<float> pv, V3<float> pw) {
    const V3<float> u = add_f(vel, cross_f(om, r));
    const V3<float> v = sub_f(u, D.other(u));
    const float vn = dot_f(n, v);
    const V3<float> vt = axpy_f(-vn, n, v);
    const float fn = lambda_n / h;
    const float x1 = __fmul_rn(mud, fabsf(fn)), x2 = sqrtf(dot_f(vt, vt));
    float fact = (x1 < x2) ? x1 : x2;
    V3<float> dv = v3<float>(0.f, 0.f, 0.f);
    if (vt.x != 0.f || vt.y != 0.f || vt.z != 0.f) dv = scale_f(-fact, v3<float>(vt.x / x2, vt.y / x2, vt.z / x2));
    const V3<float> ut = add_f(pv, cross_f(pw, r));
    const float vntil = dot_f(n, sub_f(ut, D.other(ut)));
    const float m = __fmul_rn(-e, vntil);
    fact = __fadd_rn(-vn, (m < 0.f) ? m : 0.f);
    dv = axpy_f(fact, n, dv);
    const V3<float> c = cross_f(r, n);
    const float w = __fadd_rn(invm, dot_f(c, mulv_f(I, c)));
    const V3<float> P = scale_f(1.0f / __fadd_rn(w, D.other(w)), dv);
    if (!fixed) {
        vel = D.side ? add_f(vel, scale_f(invm, P)) : axpy_f(invm, P, vel);
        om = add_f(om, mulv_f(I, cross_f(r, P)));
    }
}

}  // namespace rp
