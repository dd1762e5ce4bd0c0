// Reverse-mode derivative of the XPBD substep (the adjoint of pbd_simulate_with_constraints,
// src/physics/pbd.cpp:468-747): free bodies under gravity, the external joints (positional, mutual
// orientation, hinge, spherical, with limits) and, with collisions enabled, hull-hull contacts
// (GJK/EPA normal, clipped manifold, normal and static-friction solve, velocity solver with dynamic
// friction and restitution; rp_adjoint_contact.cuh).
//
// The forward substep is written once, templated on its scalar type S: with S = double it reproduces the
// all-FP64 step (same operations in the same order, built without FMA contraction) and runs the trajectory
// and its checkpoints; with S = AVar every vector operation also appends (parent, partial derivative) edges
// to the worker's tape, and the tape swept backwards turns the adjoint of a substep's end state into the
// adjoint of its start state. Trajectories are checkpointed every K frames; the backward pass recomputes
// each K-frame segment from its checkpoint (the last one is still there from the forward pass), keeping the
// start state of every substep and the discrete state of every frame (broad-phase pairs, awake bodies),
// then replays and reverses the substeps last to first.
//
// What is parallel: a substep's tape depends on its start state alone, so the substeps of a segment are
// taped side by side, one block each; a tape is then ordered by level (the longest path from its inputs),
// and the reverse sweep takes a level at a time, a whole block wide.
//
// Held fixed, as derivatives of discrete events: the broad-phase pair list and the set of awake
// bodies of each frame, every branch taken at a comparison (a joint limit or a contact acting or
// not, static friction holding or not, a clipping test), the support vertices and faces that GJK,
// EPA and the clipping select, and the FP32 roundings of the clipping (differentiated as identity).
#pragma once
#include <math.h>
#include "rp_math.cuh"
#include "rp_world.h"

namespace rp {

// ---------------------------------------------------------------------------------------------
// Tape of one substep: entries (values with derivatives) numbered in the order they are made, with their
// level (0 for an input, else one more than the highest of its parents'), and the edges to their parents.
// An edge whose partial derivative is zero, or whose parent is a constant, is not written, and an entry
// without edges is a constant.
struct Tape {
    int2* edge;        // parent, child
    double* partial;   // d child / d parent
    int* level;        // [ncap]
    int n, m, ncap, mcap, levels, overflow;
};

__shared__ Tape s_tape;   // one thread of a block tapes

struct AVar {
    double v;
    int id, lev;       // tape entry (-1 for a constant) and its level
    __device__ AVar() : v(0.0), id(-1), lev(-1) {}
    __device__ AVar(double x) : v(x), id(-1), lev(-1) {}
    __device__ AVar(double x, int i, int l) : v(x), id(i), lev(l) {}
};

// the value v with K edges
template <int K>
__device__ __forceinline__ AVar a_push(double v, const int (&id)[K], const int (&lv)[K], const double (&d)[K]) {
    const Tape t = s_tape;
    if (t.n >= t.ncap || t.m + K > t.mcap) {
        s_tape.overflow = 1;
        return AVar(v);
    }
    int m = t.m, lev = -1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        // (a zero test on the bits: GB300 issues an FP64 compare at 1/64 of the integer rate)
        if (id[k] < 0 || (__double_as_longlong(d[k]) << 1) == 0) continue;
        t.edge[m] = make_int2(id[k], t.n);
        t.partial[m] = d[k];
        lev = max(lev, lv[k]);
        ++m;
    }
    if (lev < 0) return AVar(v);
    t.level[t.n] = ++lev;
    s_tape.n = t.n + 1;
    s_tape.m = m;
    s_tape.levels = max(t.levels, lev + 1);
    return AVar(v, t.n, lev);
}

__device__ __forceinline__ AVar a_leaf(double x) {
    const int i = s_tape.n;
    if (i >= s_tape.ncap) {
        s_tape.overflow = 1;
        return AVar(x);
    }
    s_tape.level[i] = 0;
    s_tape.n = i + 1;
    s_tape.levels = max(s_tape.levels, 1);   // a tape of inputs alone (a scene of fixed bodies) has one level
    return AVar(x, i, 0);
}
__device__ __noinline__ AVar a_op1(double v, const AVar& a, double da) {
    const int id[1] = {a.id}, lv[1] = {a.lev};
    const double d[1] = {da};
    return a_push<1>(v, id, lv, d);
}
__device__ __noinline__ AVar a_op2(double v, const AVar& a, double da, const AVar& b, double db) {
    const int id[2] = {a.id, b.id}, lv[2] = {a.lev, b.lev};
    const double d[2] = {da, db};
    return a_push<2>(v, id, lv, d);
}
// s0 a0 b0 + s1 a1 b1 (+ ...), whose value v the caller formed: one entry, an edge per factor
__device__ __forceinline__ AVar a_sum2(double v, double s0, const AVar& a0, const AVar& b0, double s1, const AVar& a1, const AVar& b1) {
    const int id[4] = {a0.id, b0.id, a1.id, b1.id}, lv[4] = {a0.lev, b0.lev, a1.lev, b1.lev};
    const double d[4] = {s0 * b0.v, s0 * a0.v, s1 * b1.v, s1 * a1.v};
    return a_push<4>(v, id, lv, d);
}
__device__ __forceinline__ AVar a_sum3(double v, double s0, const AVar& a0, const AVar& b0, double s1, const AVar& a1, const AVar& b1,
                                       double s2, const AVar& a2, const AVar& b2) {
    const int id[6] = {a0.id, b0.id, a1.id, b1.id, a2.id, b2.id}, lv[6] = {a0.lev, b0.lev, a1.lev, b1.lev, a2.lev, b2.lev};
    const double d[6] = {s0 * b0.v, s0 * a0.v, s1 * b1.v, s1 * a1.v, s2 * b2.v, s2 * a2.v};
    return a_push<6>(v, id, lv, d);
}
__device__ __forceinline__ AVar a_sum4(double v, double s0, const AVar& a0, const AVar& b0, double s1, const AVar& a1, const AVar& b1,
                                       double s2, const AVar& a2, const AVar& b2, double s3, const AVar& a3, const AVar& b3) {
    const int id[8] = {a0.id, b0.id, a1.id, b1.id, a2.id, b2.id, a3.id, b3.id};
    const int lv[8] = {a0.lev, b0.lev, a1.lev, b1.lev, a2.lev, b2.lev, a3.lev, b3.lev};
    const double d[8] = {s0 * b0.v, s0 * a0.v, s1 * b1.v, s1 * a1.v, s2 * b2.v, s2 * a2.v, s3 * b3.v, s3 * a3.v};
    return a_push<8>(v, id, lv, d);
}

__device__ __forceinline__ AVar operator+(const AVar& a, const AVar& b) { return a_op2(a.v + b.v, a, 1.0, b, 1.0); }
__device__ __forceinline__ AVar operator-(const AVar& a, const AVar& b) { return a_op2(a.v - b.v, a, 1.0, b, -1.0); }
__device__ __forceinline__ AVar operator*(const AVar& a, const AVar& b) { return a_op2(a.v * b.v, a, b.v, b, a.v); }
__device__ __forceinline__ AVar operator/(const AVar& a, const AVar& b) {
    const double q = a.v / b.v, r = 1.0 / b.v;
    return a_op2(q, a, r, b, -q * r);
}
__device__ __forceinline__ AVar operator-(const AVar& a) { return a_op1(-a.v, a, -1.0); }
__device__ __forceinline__ AVar operator+(const AVar& a, double b) { return a + AVar(b); }
__device__ __forceinline__ AVar operator-(const AVar& a, double b) { return a - AVar(b); }
__device__ __forceinline__ AVar operator*(const AVar& a, double b) { return a * AVar(b); }
__device__ __forceinline__ AVar operator/(const AVar& a, double b) { return a / AVar(b); }
__device__ __forceinline__ AVar operator+(double a, const AVar& b) { return AVar(a) + b; }
__device__ __forceinline__ AVar operator-(double a, const AVar& b) { return AVar(a) - b; }
__device__ __forceinline__ AVar operator*(double a, const AVar& b) { return AVar(a) * b; }
__device__ __forceinline__ AVar operator/(double a, const AVar& b) { return AVar(a) / b; }
__device__ __forceinline__ bool operator<(const AVar& a, const AVar& b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>(const AVar& a, const AVar& b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<=(const AVar& a, const AVar& b) { return a.v <= b.v; }
__device__ __forceinline__ bool operator>=(const AVar& a, const AVar& b) { return a.v >= b.v; }
__device__ __forceinline__ bool operator==(const AVar& a, const AVar& b) { return a.v == b.v; }
__device__ __forceinline__ bool operator!=(const AVar& a, const AVar& b) { return a.v != b.v; }
__device__ __forceinline__ AVar sqrt(const AVar& a) {
    const double r = ::sqrt(a.v);
    return a_op1(r, a, r > 0.0 ? 0.5 / r : 0.0);
}
__device__ __forceinline__ AVar sin(const AVar& a) { return a_op1(::sin(a.v), a, ::cos(a.v)); }
__device__ __forceinline__ AVar cos(const AVar& a) { return a_op1(::cos(a.v), a, -::sin(a.v)); }
__device__ __forceinline__ AVar asin(const AVar& a) {
    const double s = 1.0 - a.v * a.v;
    return a_op1(::asin(a.v), a, s > 0.0 ? 1.0 / ::sqrt(s) : 0.0);
}
__device__ __forceinline__ AVar fabs(const AVar& a) { return a_op1(::fabs(a.v), a, a.v < 0.0 ? -1.0 : 1.0); }
// the clipping's float roundings (clipping.cpp:13,27,30,36): the value rounds, the derivative is 1
__device__ __forceinline__ AVar g_f32(const AVar& a) { return a_op1((double)(float)a.v, a, 1.0); }
__device__ __forceinline__ double g_f32(double a) { return (double)(float)a; }

// The vector algebra of rp_math.cuh, an entry per component: the same values in the same order of
// operations, and the products' partials straight from the operands. A scalar tape of the same step held
// about 3 times the entries.
__device__ __noinline__ V3<AVar> vadd(const V3<AVar>& a, const V3<AVar>& b) { return v3<AVar>(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __noinline__ V3<AVar> vsub(const V3<AVar>& a, const V3<AVar>& b) { return v3<AVar>(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __noinline__ V3<AVar> vscale(const AVar& s, const V3<AVar>& v) { return v3<AVar>(s * v.x, s * v.y, s * v.z); }
__device__ __noinline__ AVar vdot(const V3<AVar>& a, const V3<AVar>& b) {
    return a_sum3(a.x.v * b.x.v + a.y.v * b.y.v + a.z.v * b.z.v, 1.0, a.x, b.x, 1.0, a.y, b.y, 1.0, a.z, b.z);
}
// ab - cd
__device__ __noinline__ AVar a_cross1(const AVar& a, const AVar& b, const AVar& c, const AVar& d) {
    return a_sum2(a.v * b.v - c.v * d.v, 1.0, a, b, -1.0, c, d);
}
__device__ __forceinline__ V3<AVar> vcross(const V3<AVar>& a, const V3<AVar>& b) {
    return v3<AVar>(a_cross1(a.y, b.z, a.z, b.y), a_cross1(a.z, b.x, a.x, b.z), a_cross1(a.x, b.y, a.y, b.x));
}
__device__ __noinline__ AVar vlen(const V3<AVar>& v) {
    const double l = ::sqrt(v.x.v * v.x.v + v.y.v * v.y.v + v.z.v * v.z.v), r = l > 0.0 ? 1.0 / l : 0.0;
    const int id[3] = {v.x.id, v.y.id, v.z.id}, lv[3] = {v.x.lev, v.y.lev, v.z.lev};
    const double d[3] = {v.x.v * r, v.y.v * r, v.z.v * r};
    return a_push<3>(l, id, lv, d);
}
__device__ __noinline__ V3<AVar> vnorm(const V3<AVar>& v) {
    if (!(v.x.v != 0.0 || v.y.v != 0.0 || v.z.v != 0.0)) return v3<AVar>(AVar(0.0), AVar(0.0), AVar(0.0));
    const double l = ::sqrt(v.x.v * v.x.v + v.y.v * v.y.v + v.z.v * v.z.v), r = 1.0 / l;
    const double x = v.x.v / l, y = v.y.v / l, z = v.z.v / l;
    const int id[3] = {v.x.id, v.y.id, v.z.id}, lv[3] = {v.x.lev, v.y.lev, v.z.lev};
    const double dx[3] = {(1.0 - x * x) * r, -x * y * r, -x * z * r}, dy[3] = {-x * y * r, (1.0 - y * y) * r, -y * z * r},
                 dz[3] = {-x * z * r, -y * z * r, (1.0 - z * z) * r};
    return v3<AVar>(a_push<3>(x, id, lv, dx), a_push<3>(y, id, lv, dy), a_push<3>(z, id, lv, dz));
}
// v / c
__device__ __forceinline__ V3<double> g_div(const V3<double>& v, double c) { return v3<double>(v.x / c, v.y / c, v.z / c); }
__device__ __noinline__ V3<AVar> g_div(const V3<AVar>& v, const AVar& c) {
    const double r = 1.0 / c.v, x = v.x.v / c.v, y = v.y.v / c.v, z = v.z.v / c.v;
    return v3<AVar>(a_op2(x, v.x, r, c, -x * r), a_op2(y, v.y, r, c, -y * r), a_op2(z, v.z, r, c, -z * r));
}
__device__ __noinline__ Qt<AVar> qmul(const Qt<AVar>& a, const Qt<AVar>& b) {
    Qt<AVar> r;
    r.w = a_sum4(a.w.v * b.w.v - a.x.v * b.x.v - a.y.v * b.y.v - a.z.v * b.z.v, 1.0, a.w, b.w, -1.0, a.x, b.x, -1.0, a.y, b.y, -1.0, a.z, b.z);
    r.x = a_sum4(a.w.v * b.x.v + a.x.v * b.w.v + a.y.v * b.z.v - a.z.v * b.y.v, 1.0, a.w, b.x, 1.0, a.x, b.w, 1.0, a.y, b.z, -1.0, a.z, b.y);
    r.y = a_sum4(a.w.v * b.y.v + a.y.v * b.w.v + a.z.v * b.x.v - a.x.v * b.z.v, 1.0, a.w, b.y, 1.0, a.y, b.w, 1.0, a.z, b.x, -1.0, a.x, b.z);
    r.z = a_sum4(a.w.v * b.z.v + a.z.v * b.w.v + a.x.v * b.y.v - a.y.v * b.x.v, 1.0, a.w, b.z, 1.0, a.z, b.w, 1.0, a.x, b.y, -1.0, a.y, b.x);
    return r;
}
__device__ __noinline__ Qt<AVar> qnormalize(const Qt<AVar>& q) {
    const double l = ::sqrt(q.x.v * q.x.v + q.y.v * q.y.v + q.z.v * q.z.v + q.w.v * q.w.v), r = 1.0 / l;
    const double u[4] = {q.x.v / l, q.y.v / l, q.z.v / l, q.w.v / l};
    const int id[4] = {q.x.id, q.y.id, q.z.id, q.w.id}, lv[4] = {q.x.lev, q.y.lev, q.z.lev, q.w.lev};
    AVar o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        double d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] = ((i == j ? 1.0 : 0.0) - u[i] * u[j]) * r;
        o[i] = a_push<4>(u[i], id, lv, d);
    }
    return qt<AVar>(o[0], o[1], o[2], o[3]);
}
// a row of qrotate's first product, q.w v_i + q_j v_k - q_k v_j, and of its second,
// i_i q.w - iw q_i - i_j q_k + i_k q_j
__device__ __noinline__ AVar a_rot1(const AVar& qw, const AVar& vi, const AVar& qj, const AVar& vk, const AVar& qk, const AVar& vj) {
    return a_sum3(qw.v * vi.v + qj.v * vk.v - qk.v * vj.v, 1.0, qw, vi, 1.0, qj, vk, -1.0, qk, vj);
}
__device__ __noinline__ AVar a_rot2(const AVar& ii, const AVar& qw, const AVar& iw, const AVar& qi, const AVar& ij, const AVar& qk,
                                    const AVar& ik, const AVar& qj) {
    return a_sum4((ii.v * qw.v) + (iw.v * -qi.v) + (ij.v * -qk.v) - (ik.v * -qj.v), 1.0, ii, qw, -1.0, iw, qi, -1.0, ij, qk, 1.0, ik, qj);
}
__device__ __noinline__ V3<AVar> qrotate(const Qt<AVar>& q, const V3<AVar>& v) {
    const AVar ix = a_rot1(q.w, v.x, q.y, v.z, q.z, v.y), iy = a_rot1(q.w, v.y, q.z, v.x, q.x, v.z), iz = a_rot1(q.w, v.z, q.x, v.y, q.y, v.x);
    const AVar iw = a_sum3(-q.x.v * v.x.v - q.y.v * v.y.v - q.z.v * v.z.v, -1.0, q.x, v.x, -1.0, q.y, v.y, -1.0, q.z, v.z);
    return v3<AVar>(a_rot2(ix, q.w, iw, q.x, iy, q.z, iz, q.y), a_rot2(iy, q.w, iw, q.y, iz, q.x, ix, q.z),
                    a_rot2(iz, q.w, iw, q.z, ix, q.y, iy, q.x));
}
__device__ __forceinline__ AVar a_diag(const AVar& a, const AVar& b) {   // 1 - 2 a a - 2 b b
    const int id[2] = {a.id, b.id}, lv[2] = {a.lev, b.lev};
    const double d[2] = {-4.0 * a.v, -4.0 * b.v};
    return a_push<2>(1.0 - 2.0 * a.v * a.v - 2.0 * b.v * b.v, id, lv, d);
}
__device__ __noinline__ AVar a_off(const AVar& a, const AVar& b, double s, const AVar& c, const AVar& d) {   // 2 a b + s 2 c d, s = +-1
    const double p = 2.0 * a.v * b.v, q = 2.0 * c.v * d.v;
    return a_sum2(s > 0.0 ? p + q : p - q, 2.0, a, b, 2.0 * s, c, d);
}
__device__ __noinline__ M3<AVar> qmat3(const Qt<AVar>& q) {
    M3<AVar> r;
    r.d[0][0] = a_diag(q.y, q.z);
    r.d[1][1] = a_diag(q.x, q.z);
    r.d[2][2] = a_diag(q.x, q.y);
    r.d[1][0] = a_off(q.x, q.y, 1.0, q.w, q.z);
    r.d[2][0] = a_off(q.x, q.z, -1.0, q.w, q.y);
    r.d[0][1] = a_off(q.x, q.y, -1.0, q.w, q.z);
    r.d[2][1] = a_off(q.y, q.z, 1.0, q.w, q.x);
    r.d[0][2] = a_off(q.x, q.z, 1.0, q.w, q.y);
    r.d[1][2] = a_off(q.y, q.z, -1.0, q.w, q.x);
    return r;
}
__device__ __noinline__ AVar a_row(const AVar& a0, const AVar& b0, const AVar& a1, const AVar& b1, const AVar& a2, const AVar& b2) {
    return a_sum3(a0.v * b0.v + a1.v * b1.v + a2.v * b2.v, 1.0, a0, b0, 1.0, a1, b1, 1.0, a2, b2);
}
__device__ __noinline__ V3<AVar> mmulv(const M3<AVar>& m, const V3<AVar>& v) {
    return v3<AVar>(a_row(m.d[0][0], v.x, m.d[0][1], v.y, m.d[0][2], v.z), a_row(m.d[1][0], v.x, m.d[1][1], v.y, m.d[1][2], v.z),
                    a_row(m.d[2][0], v.x, m.d[2][1], v.y, m.d[2][2], v.z));
}
__device__ __noinline__ M3<AVar> world_tensor(const Qt<AVar>& q, const M3<AVar>& local) {
    const M3<AVar> r = qmat3(q);
    M3<AVar> aux, o;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) aux.d[i][j] = a_row(r.d[i][0], local.d[0][j], r.d[i][1], local.d[1][j], r.d[i][2], local.d[2][j]);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) o.d[i][j] = a_row(aux.d[i][0], r.d[j][0], aux.d[i][1], r.d[j][1], aux.d[i][2], r.d[j][2]);
    return o;
}

// the scalar pass calls the same names on doubles
__device__ __forceinline__ double sqrt(double a) { return ::sqrt(a); }
__device__ __forceinline__ double sin(double a) { return ::sin(a); }
__device__ __forceinline__ double cos(double a) { return ::cos(a); }
__device__ __forceinline__ double asin(double a) { return ::asin(a); }
__device__ __forceinline__ double fabs(double a) { return ::fabs(a); }

template <> struct Tiny<AVar> { static constexpr double v = 1e-50; };
__device__ __forceinline__ double val(double x) { return x; }
__device__ __forceinline__ double val(const AVar& x) { return x.v; }
template <typename S> __device__ __forceinline__ V3<double> vval(const V3<S>& a) { return v3<double>(val(a.x), val(a.y), val(a.z)); }

// ---------------------------------------------------------------------------------------------
// The substep on bodies held in registers (mirrors rp_solve.cuh's all-FP64 path term for term)
template <typename S>
struct GBody {
    V3<S> x, px;       // position, position at the substep start
    Qt<S> q, pq;       // orientation, orientation at the substep start
    V3<S> v, w;        // velocities
    V3<S> pv, pw;      // velocities before the velocity update (previous_linear/angular_velocity)
    S invm;
    M3<S> Iinv, I;     // local inverse inertia and inertia
    S mus, mud, rest;  // static and dynamic friction, restitution
    bool fixed, active;
};

template <typename S>
__device__ __forceinline__ void g_qadd(Qt<S>& q, Qt<S> d, double s) {
    q.x = q.x + s * d.x; q.y = q.y + s * d.y; q.z = q.z + s * d.z; q.w = q.w + s * d.w;
    q = qnormalize(q);
}

// predict (pbd.cpp:537-577) with the caller's force F and no torque
template <typename S>
__device__ __noinline__ void g_predict(GBody<S>& B, V3<S> F, double h) {
    B.px = B.x;
    B.pq = B.q;
    if (B.fixed || !B.active) return;
    const V3<S> T = v3<S>(S(0.0), S(0.0), S(0.0));
    B.v = vadd(B.v, vscale(S(h) * B.invm, F));
    B.x = vadd(B.x, vscale(S(h), B.v));
    const M3<S> Iinv = world_tensor(B.q, B.Iinv), I = world_tensor(B.q, B.I);
    B.w = vadd(B.w, vscale(S(h), mmulv(Iinv, vsub(T, vcross(B.w, mmulv(I, B.w))))));
    const Qt<S> qd = qmul(qt<S>(B.w.x, B.w.y, B.w.z, S(0.0)), B.q);
    B.q.x = B.q.x + h * 0.5 * qd.x; B.q.y = B.q.y + h * 0.5 * qd.y;
    B.q.z = B.q.z + h * 0.5 * qd.z; B.q.w = B.q.w + h * 0.5 * qd.w;
    B.q = qnormalize(B.q);
}

// velocity update (pbd.cpp:623-643)
template <typename S>
__device__ void g_velocity(GBody<S>& B, double h) {
    if (B.fixed || !B.active) return;
    B.pv = B.v;
    B.pw = B.w;
    const V3<S> dx = vsub(B.x, B.px);
    B.v = vscale(S(1.0 / h), dx);
    const Qt<S> dq = qmul(B.q, qinverse(B.pq));
    B.w = (val(dq.w) >= 0.0) ? vscale(S(2.0 / h), v3<S>(dq.x, dq.y, dq.z)) : vscale(S(-2.0 / h), v3<S>(dq.x, dq.y, dq.z));
}

template <typename S> struct GPcpd { V3<S> r1, r2; M3<S> I1, I2; };

template <typename S>
__device__ __forceinline__ GPcpd<S> g_pcpd(const GBody<S>& a, const GBody<S>& b, V3<S> r1, V3<S> r2) {
    GPcpd<S> p;
    p.r1 = qrotate(a.q, r1);
    p.r2 = qrotate(b.q, r2);
    p.I1 = world_tensor(a.q, a.Iinv);
    p.I2 = world_tensor(b.q, b.Iinv);
    return p;
}

template <typename S>
__device__ S g_pos_dlambda(const GBody<S>& a, const GBody<S>& b, const GPcpd<S>& p, double h, double compliance, S lambda, V3<S> dx) {
    const S c = vlen(dx);
    if (c <= Tiny<S>::v) return S(0.0);
    const V3<S> n = g_div(dx, c);
    const S w1 = a.invm + vdot(vcross(p.r1, n), mmulv(p.I1, vcross(p.r1, n)));
    const S w2 = b.invm + vdot(vcross(p.r2, n), mmulv(p.I2, vcross(p.r2, n)));
    const S til = S(compliance) / (S(h) * S(h));
    return (-c - til * lambda) / (w1 + w2 + til);
}

template <typename S>
__device__ void g_pos_apply(GBody<S>& a, GBody<S>& b, const GPcpd<S>& p, S dl, V3<S> dx) {
    const S c = vlen(dx);
    if (c <= Tiny<S>::v) return;
    const V3<S> n = g_div(dx, c);
    const V3<S> imp = vscale(dl, n);
    if (!a.fixed) a.x = vadd(a.x, vscale(a.invm, imp));
    if (!b.fixed) b.x = vadd(b.x, vscale(-b.invm, imp));
    const V3<S> a1 = mmulv(p.I1, vcross(p.r1, imp));
    const V3<S> a2 = mmulv(p.I2, vcross(p.r2, imp));
    const Qt<S> q1 = qmul(qt<S>(a1.x, a1.y, a1.z, S(0.0)), a.q);
    const Qt<S> q2 = qmul(qt<S>(a2.x, a2.y, a2.z, S(0.0)), b.q);
    if (!a.fixed) g_qadd(a.q, q1, 0.5);
    if (!b.fixed) g_qadd(b.q, q2, -0.5);
}

template <typename S> struct GAcpd { M3<S> I1, I2; };

template <typename S>
__device__ __forceinline__ GAcpd<S> g_acpd(const GBody<S>& a, const GBody<S>& b) {
    GAcpd<S> r;
    r.I1 = world_tensor(a.q, a.Iinv);
    r.I2 = world_tensor(b.q, b.Iinv);
    return r;
}

template <typename S>
__device__ S g_ang_dlambda(const GAcpd<S>& A, double h, double compliance, S lambda, V3<S> dq) {
    const S th = vlen(dq);
    if (th <= Tiny<S>::v) return S(0.0);
    const V3<S> n = g_div(dq, th);
    const S w1 = vdot(n, mmulv(A.I1, n));
    const S w2 = vdot(n, mmulv(A.I2, n));
    const S til = S(compliance) / (S(h) * S(h));
    return (-th - til * lambda) / (w1 + w2 + til);
}

template <typename S>
__device__ void g_ang_apply(GBody<S>& a, GBody<S>& b, const GAcpd<S>& A, S dl, V3<S> dq) {
    const S th = vlen(dq);
    if (th <= Tiny<S>::v) return;
    const V3<S> n = g_div(dq, th);
    const V3<S> imp = vscale(-dl, n);
    const V3<S> a1 = mmulv(A.I1, imp);
    const V3<S> a2 = mmulv(A.I2, imp);
    const Qt<S> q1 = qmul(qt<S>(a1.x, a1.y, a1.z, S(0.0)), a.q);
    const Qt<S> q2 = qmul(qt<S>(a2.x, a2.y, a2.z, S(0.0)), b.q);
    if (!a.fixed) g_qadd(a.q, q1, 0.5);
    if (!b.fixed) g_qadd(b.q, q2, -0.5);
}

template <typename S>
__device__ bool g_limit_angle(V3<S> n, V3<S> n1, V3<S> n2, double alpha, double beta, V3<S>& dq) {
    const S pi = S(3.14159265358979);
    S phi = asin(vdot(vcross(n1, n2), n));
    if (vdot(n1, n2) < S(0.0)) phi = pi - phi;
    if (phi > pi) phi = phi - S(2.0) * pi;
    if (phi < -pi) phi = phi + S(2.0) * pi;
    if (phi < S(alpha) || phi > S(beta)) {
        phi = (phi > S(beta)) ? S(beta) : ((phi < S(alpha)) ? S(alpha) : phi);
        V3<S> ax = n;
        if (vlen(ax) != S(0.0)) ax = vnorm(ax);
        const S s = sin(phi / S(2.0));
        const Qt<S> rot = qt<S>(ax.x * s, ax.y * s, ax.z * s, cos(phi / S(2.0)));
        n1 = qrotate(rot, n1);
        dq = vcross(n1, n2);
        return true;
    }
    return false;
}

template <typename S>
__device__ void g_angle_correction(GBody<S>& a, GBody<S>& b, V3<S> dq, double h, S& lam) {
    const GAcpd<S> A = g_acpd(a, b);
    const S d2 = g_ang_dlambda(A, h, 0.0, lam, dq);
    g_ang_apply(a, b, A, d2, dq);
    lam = lam + d2;
}

// one external constraint (pbd.cpp:81-379); lam: its 4 per-substep lambdas
template <typename S>
__device__ __noinline__ void g_ext_solve(GBody<S>& a, GBody<S>& b, const ExtConstraint& C, S* lam, double h) {
    const V3<S> r1 = v3<S>(S(C.r1[0]), S(C.r1[1]), S(C.r1[2])), r2 = v3<S>(S(C.r2[0]), S(C.r2[1]), S(C.r2[2]));
    auto anchor = [&](const GPcpd<S>& p) { return vsub(vadd(a.x, p.r1), vadd(b.x, p.r2)); };
    switch (C.type) {
    case CON_POSITIONAL: {
        const V3<S> dx = vsub(vsub(a.x, b.x), v3<S>(S(C.distance[0]), S(C.distance[1]), S(C.distance[2])));
        const GPcpd<S> p = g_pcpd(a, b, r1, r2);
        const S dl = g_pos_dlambda(a, b, p, h, C.compliance, lam[0], dx);
        g_pos_apply(a, b, p, dl, dx);
        lam[0] = lam[0] + dl;
    } break;
    case CON_MUTUAL_ORIENTATION: {
        const GAcpd<S> A = g_acpd(a, b);
        const Qt<S> aux = qmul(a.q, qinverse(b.q));
        const V3<S> dq = v3<S>(S(2.0) * aux.x, S(2.0) * aux.y, S(2.0) * aux.z);
        const S dl = g_ang_dlambda(A, h, C.compliance, lam[0], dq);
        g_ang_apply(a, b, A, dl, dq);
        lam[0] = lam[0] + dl;
    } break;
    case CON_HINGE: {
        const GAcpd<S> A = g_acpd(a, b);
        const V3<S> dq = vcross(qaxis(a.q, C.a1), qaxis(b.q, C.a2));
        S dl = g_ang_dlambda(A, h, C.compliance, lam[1], dq);
        g_ang_apply(a, b, A, dl, dq);
        lam[1] = lam[1] + dl;
        const GPcpd<S> p = g_pcpd(a, b, r1, r2);
        const V3<S> dx = anchor(p);
        dl = g_pos_dlambda(a, b, p, h, 0.0, lam[0], dx);
        g_pos_apply(a, b, p, dl, dx);
        lam[0] = lam[0] + dl;
        if (C.limited) {
            V3<S> dq2;
            if (g_limit_angle(qaxis(a.q, C.a1), qaxis(a.q, C.l1), qaxis(b.q, C.l2), C.lo, C.hi, dq2))
                g_angle_correction(a, b, dq2, h, lam[2]);
        }
    } break;
    case CON_SPHERICAL: {
        const GPcpd<S> p = g_pcpd(a, b, r1, r2);
        const V3<S> dx = anchor(p);
        const S dl = g_pos_dlambda(a, b, p, h, 0.0, lam[0], dx);
        g_pos_apply(a, b, p, dl, dx);
        lam[0] = lam[0] + dl;
        const double EPS64 = 1e-50;
        {
            const V3<S> n1 = qaxis(a.q, C.a1), n2 = qaxis(b.q, C.a2);
            V3<S> n = vcross(n1, n2);
            const S nl = vlen(n);
            if (val(nl) > EPS64) {
                n = g_div(n, nl);
                V3<S> dq2;
                if (g_limit_angle(n, n1, n2, C.lo, C.hi, dq2)) g_angle_correction(a, b, dq2, h, lam[1]);
            }
        }
        {
            const V3<S> a1 = qaxis(a.q, C.a1), b1 = qaxis(a.q, C.l1), a2 = qaxis(b.q, C.a2), b2 = qaxis(b.q, C.l2);
            V3<S> n = vadd(a1, a2);
            const S nl = vlen(n);
            if (val(nl) > EPS64) {
                n = g_div(n, nl);
                V3<S> n1 = vsub(b1, vscale(vdot(n, b1), n)), n2 = vsub(b2, vscale(vdot(n, b2), n));
                const S l1 = vlen(n1), l2 = vlen(n2);
                if (val(l1) > EPS64 && val(l2) > EPS64) {
                    n1 = g_div(n1, l1);
                    n2 = g_div(n2, l2);
                    V3<S> dq2;
                    if (g_limit_angle(n, n1, n2, C.lo2, C.hi2, dq2)) g_angle_correction(a, b, dq2, h, lam[2]);
                }
            }
        }
    } break;
    default: break;
    }
}

}  // namespace rp
