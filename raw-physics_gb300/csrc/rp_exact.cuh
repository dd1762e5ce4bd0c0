// The all-FP64 solves with eight lanes a solver node: four per body, three of them a vector component (or a
// matrix row) each and the fourth a quaternion's w (Oct).
//
// GB300 issues one FP64 warp instruction per SM sub-partition in 64 cycles, whatever the number of active
// lanes and however independent the instructions are; a division or square root is ten of them. An FP64
// solve's time is therefore the number of FP64 instructions of its warp, and a vector operation costs a
// third when three lanes compute a component each and exchange them (a 64-bit shuffle takes 24 cycles).
// A contact of the position sweep takes 190 to 320 such instructions instead of about 1000 with a lane per
// body, a contact of the velocity sweep 95 instead of 200, a predict step 130 instead of 420. A warp with a lane per
// body would do 16 nodes at that price, but a scene's levels are mostly a few nodes wide: 2048 scenes of up to 512
// bodies, which keep every FP64 unit busy, 1112 -> 541 ms a frame, 64 scenes 342 -> 84, 12000 bodies in one scene 185 ->
// 49. (Wide levels, as the coloured order has, get a CTA: make_view.) Every component is formed by the reference's own
// expression in its order of operations, so the results are bit for bit those of the serial solve.
//
// All lanes of a body hold its whole pose and every vector; what is spread over them is the arithmetic.
// As with a lane per body (Duo), the second body's lanes work on negated vectors.
//
// References (raw-physics): pbd.cpp:81-406 (solves), :646-711 (velocity solver);
// pbd_base_constraints.cpp:6-227; physics_util.cpp:26-63.
#pragma once
#include "rp_solve.cuh"

namespace rp {

struct Oct {
    unsigned oct, quad;   // the node's lanes, the body's lanes
    int side, c;          // 0: the node's first body, 1: its second; this lane's component
    __device__ __forceinline__ double other(double v) const { return __shfl_xor_sync(oct, v, 4); }
    __device__ __forceinline__ V3<double> other(V3<double> v) const { return v3<double>(other(v.x), other(v.y), other(v.z)); }
    __device__ __forceinline__ Qt<double> other(Qt<double> q) const { return qt<double>(other(q.x), other(q.y), other(q.z), other(q.w)); }
    // every lane's component to all lanes of the body
    __device__ __forceinline__ V3<double> all(double v) const {
        return v3<double>(__shfl_sync(quad, v, 0, 4), __shfl_sync(quad, v, 1, 4), __shfl_sync(quad, v, 2, 4));
    }
    __device__ __forceinline__ Qt<double> all4(double v) const {
        return qt<double>(__shfl_sync(quad, v, 0, 4), __shfl_sync(quad, v, 1, 4), __shfl_sync(quad, v, 2, 4), __shfl_sync(quad, v, 3, 4));
    }
    // this lane's component and the two after it in cyclic order (the fourth lane's are never used)
    template <typename V> __device__ __forceinline__ double at(const V& v) const { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }
    template <typename V> __device__ __forceinline__ double at1(const V& v) const { return c == 0 ? v.y : (c == 1 ? v.z : v.x); }
    template <typename V> __device__ __forceinline__ double at2(const V& v) const { return c == 0 ? v.z : (c == 1 ? v.x : v.y); }
    __device__ __forceinline__ double at4(const Qt<double>& q) const { return c == 3 ? q.w : at(q); }
    template <typename V> __device__ __forceinline__ V own(const V& v) const { return side ? v3<double>(-v.x, -v.y, -v.z) : v; }
    template <typename V> __device__ __forceinline__ V first(const V& mine, const V& theirs) const { return side ? theirs : mine; }
    template <typename V> __device__ __forceinline__ V second(const V& mine, const V& theirs) const { return side ? mine : theirs; }
    __device__ __forceinline__ bool lead() const { return side == 0 && c == 0; }

    // components of a x b, of a matrix row times v; sums of three components
    __device__ __forceinline__ double cross(const V3<double>& a, const V3<double>& b) const { return at1(a) * at2(b) - at2(a) * at1(b); }
    __device__ __forceinline__ double row(const V3<double>& m, const V3<double>& v) const { return m.x * v.x + m.y * v.y + m.z * v.z; }
    __device__ __forceinline__ double dot(double a, double b) const {
        const V3<double> p = all(a * b);
        return p.x + p.y + p.z;
    }
    // qrotate
    __device__ __forceinline__ V3<double> rotate(const Qt<double>& q, const V3<double>& v) const {
        const bool w = c == 3;
        const double i = (w ? -q.x : q.w) * (w ? v.x : at(v)) + (w ? -q.y : at1(q)) * (w ? v.y : at2(v)) -
                         (w ? q.z : at2(q)) * (w ? v.z : at1(v));
        const Qt<double> t = all4(i);
        return all((at(t) * q.w) + (t.w * -at(q)) + (at1(t) * -at2(q)) - (at2(t) * -at1(q)));
    }
    // this lane's component of a b
    __device__ __forceinline__ double mul(const Qt<double>& a, const Qt<double>& b) const {
        const bool w = c == 3;
        return a.w * at4(b) + (w ? -a.x : at(a)) * (w ? b.x : b.w) + (w ? -a.y : at1(a)) * (w ? b.y : at2(b)) -
               (w ? a.z : at2(a)) * (w ? b.z : at1(b));
    }
    // qnormalize of the quaternion whose component is v
    __device__ __forceinline__ Qt<double> normalize(double v) const {
        const Qt<double> s = all4(v * v);
        const double l = ::sqrt(s.x + s.y + s.z + s.w);
        return all4(v / l);
    }
    // |v|, and v / |v| when the length is above the reference's threshold
    __device__ __forceinline__ bool unit(const V3<double>& v, double& len, V3<double>& n) const {
        const double m = at(v);
        const V3<double> s = all(m * m);
        len = ::sqrt(s.x + s.y + s.z);
        if (len <= Tiny<double>::v) return false;
        n = all(m / len);
        return true;
    }
    __device__ __forceinline__ double length(const V3<double>& v) const {
        const double m = at(v);
        const V3<double> s = all(m * m);
        return ::sqrt(s.x + s.y + s.z);
    }
    // qmat3 of q: this lane's row, and the diagonals of all rows from the main one on in cyclic order. Row c from
    // its diagonal element on: 1 - 2 q_j q_j - 2 q_k q_k, 2 q_c q_c+1 - 2 w q_c+2, 2 q_c q_c+2 + 2 w q_c+1.
    struct Rot { V3<double> m, D0, D1, D2; };
    __device__ __forceinline__ Rot matrix(const Qt<double>& q) const {
        const Qt<double> d = all4(2.0 * at4(q));
        const double j = c == 0 ? q.y : q.x, dj = c == 0 ? d.y : d.x, k = c == 2 ? q.y : q.z, dk = c == 2 ? d.y : d.z;
        const double r0 = 1.0 - dj * j - dk * k, r1 = at(d) * at1(q) - d.w * at2(q), r2 = at(d) * at2(q) + d.w * at1(q);
        Rot R;
        R.D0 = all(r0);
        R.D1 = all(r1);
        R.D2 = all(r2);
        R.m = c == 0 ? v3<double>(r0, r1, r2) : (c == 1 ? v3<double>(r2, r0, r1) : v3<double>(r1, r2, r0));
        return R;
    }
    // this lane's row of world_tensor
    __device__ __forceinline__ V3<double> tensor(const Rot& R, const double (&L)[6]) const {
        const V3<double>&m = R.m, &D0 = R.D0, &D1 = R.D1, &D2 = R.D2;
        const V3<double> a = v3<double>(m.x * L[0] + m.y * L[3] + m.z * L[4], m.x * L[3] + m.y * L[1] + m.z * L[5],
                                        m.x * L[4] + m.y * L[5] + m.z * L[2]);
        return v3<double>(a.x * D0.x + a.y * D1.x + a.z * D2.x, a.x * D2.y + a.y * D0.y + a.z * D1.y,
                          a.x * D1.z + a.y * D2.z + a.z * D0.z);
    }
    __device__ __forceinline__ V3<double> tensor(const Qt<double>& q, const double (&L)[6]) const { return tensor(matrix(q), L); }
    // qaxis: the row of axis k >> 1, with -w for a negative axis
    __device__ __forceinline__ V3<double> axis(const Qt<double>& q, int k) const {
        const int a = k >> 1, rel = (c + 3 - a) % 3;   // (of the fourth lane: not used)
        const double w = k & 1 ? q.w : -q.w, qa = a == 0 ? q.x : (a == 1 ? q.y : q.z);
        const double j = a == 0 ? q.y : q.x, m = a == 2 ? q.y : q.z;
        // the third component of {a, c}: a + 2 for c = a + 1 and a + 1 for c = a + 2
        const int t = rel == 1 ? (a + 2) % 3 : (a + 1) % 3;
        const double o = t == 0 ? q.x : (t == 1 ? q.y : q.z);
        const double p = (2.0 * (rel == 0 ? j : qa)) * (rel == 0 ? j : at(q));
        const double s = (2.0 * (rel == 0 ? m : (rel == 1 ? w : -w))) * (rel == 0 ? m : o);
        return all((rel == 0 ? 1.0 - p : p) - s);
    }
};

__device__ __forceinline__ Oct oct_of_lane() {
    const unsigned lane = threadIdx.x & 31u;
    return Oct{0xffu << (lane & 24u), 0xfu << (lane & 28u), (int)((lane >> 2) & 1u), (int)(lane & 3u)};
}

// a body during a node's solves, in all of its lanes
struct OctBody {
    V3<double> x;
    Qt<double> q;
    double invm, L[6];   // local inverse inertia (xx yy zz xy xz yz)
    V3<double> I;        // this lane's row of the world inverse inertia at orientation q, while fresh
    bool fixed, fresh;
    int idx;
};

__device__ __forceinline__ OctBody load_oct(const WorldView<double>& W, int b) {
    OctBody B;
    const double4_32a p = W.pos[b], q = W.rot[b];
    B.x = v3<double>(p.x, p.y, p.z);
    B.q = qt<double>(q.x, q.y, q.z, q.w);
    B.invm = W.inv_mass[b];
#pragma unroll
    for (int i = 0; i < 6; ++i) B.L[i] = W.inv_inertia[6 * b + i];
    B.I = v3<double>(0.0, 0.0, 0.0);
    B.fixed = W.fixed[b] != 0;
    B.fresh = false;
    B.idx = b;
    return B;
}
__device__ __forceinline__ void store_oct(const WorldView<double>& W, const Oct& O, const OctBody& B) {
    if (B.fixed || O.c != 0) return;
    W.pos[B.idx] = make_double4_32a(B.x.x, B.x.y, B.x.z, 0.0);
    W.rot[B.idx] = make_double4_32a(B.q.x, B.q.y, B.q.z, B.q.w);
}
__device__ __forceinline__ void refresh(const Oct& O, OctBody& B) {
    if (!B.fresh) B.I = O.tensor(B.q, B.L);
    B.fresh = true;
}

// Positional corrections (pbd_base_constraints.cpp:6-123): dx = len n, the separation seen from this body; r its
// anchor in world axes. (With zero compliance the reference's terms in it are exact zeros.)
__device__ __forceinline__ double pos_dlambda(const Oct& O, const OctBody& B, V3<double> r, double h, double compliance, double lambda,
                                              double len, V3<double> n) {
    const double a = O.cross(r, n);
    const double w = B.invm + O.dot(a, O.row(B.I, O.all(a)));
    if (compliance == 0.0) return -len / (w + O.other(w));
    const double til = compliance / (h * h);
    return (-len - til * lambda) / (w + O.other(w) + til);
}
__device__ __forceinline__ void turn(const Oct& O, OctBody& B, double a) {
    const V3<double> t = O.all(a);
    const double dq = O.mul(qt<double>(t.x, t.y, t.z, 0.0), B.q);
    if (B.fixed) return;
    B.q = O.normalize(O.at4(B.q) + 0.5 * dq);
    B.fresh = false;
}
__device__ __forceinline__ void pos_apply(const Oct& O, OctBody& B, V3<double> r, double dl, V3<double> n) {
    const double imp = dl * O.at(n);
    turn(O, B, O.row(B.I, O.all(O.cross(r, O.all(imp)))));
    if (!B.fixed) B.x = O.all(O.at(B.x) + B.invm * imp);
}
// Angular corrections (pbd_base_constraints.cpp:125-227): dq = len n seen from this body
__device__ __forceinline__ double ang_dlambda(const Oct& O, const OctBody& B, double h, double compliance, double lambda, double len,
                                              V3<double> n) {
    const double w = O.dot(O.at(n), O.row(B.I, n));
    if (compliance == 0.0) return -len / (w + O.other(w));
    const double til = compliance / (h * h);
    return (-len - til * lambda) / (w + O.other(w) + til);
}

// collision_constraint_solve (pbd.cpp:107-154): r_lc this body's anchor, n the normal seen from it
__device__ __forceinline__ bool oct_contact(const Oct& O, OctBody& B, V3<double> r_lc, V3<double> n, double mus, V3<double> prev_x,
                                            Qt<double> prev_q, double h, double& lambda_n, double& lambda_t) {
    V3<double> r = O.rotate(B.q, r_lc);
    const double p0 = O.at(B.x) + O.at(r);
    const double d = O.dot(p0 - O.other(p0), O.at(n));
    if (!(d > 0.0)) return false;
    const V3<double> dx = O.all(d * O.at(n));
    double len, dl = 0.0;
    V3<double> u;
    const bool far = O.unit(dx, len, u);
    refresh(O, B);
    if (far) {
        dl = pos_dlambda(O, B, r, h, 0.0, lambda_n, len, u);
        pos_apply(O, B, r, dl, u);
    }
    lambda_n += dl;
    r = O.rotate(B.q, r_lc);
    refresh(O, B);
    dl = far ? pos_dlambda(O, B, r, h, 0.0, lambda_t, len, u) : 0.0;
    const double lt = lambda_t + dl;
    if (lt > mus * lambda_n) {
        // p1 - p1_til - (p2 - p2_til) with p_til from the previous pose (pbd.cpp:142-148)
        const V3<double> rp = O.rotate(prev_q, r_lc);
        const double v = (O.at(B.x) + O.at(r)) - (O.at(prev_x) + O.at(rp));
        const double dp = v - O.other(v);
        const double t = O.dot(dp, O.at(n));
        const V3<double> dt = O.all(dp - t * O.at(n));
        if (O.unit(dt, len, u)) pos_apply(O, B, r, dl, u);
        lambda_t += dl;
    }
    return true;
}

// one joint limit: the angle between n1 (first body) and n2 (second body) about n, clamped to [lo, hi]
// (limit_angle, pbd.cpp:175-217), corrected with a zero-compliance angular solve
__device__ __forceinline__ void oct_limit(const Oct& O, OctBody& B, V3<double> n, V3<double> n1, V3<double> n2, double lo, double hi,
                                          double h, double* lam) {
    if (lo <= -PI_REF && hi >= PI_REF) return;   // the wrapped angle can never leave limits at or beyond +-pi
    double phi = ::asin(O.dot(O.cross(n1, n2), O.at(n)));
    if (O.dot(O.at(n1), O.at(n2)) < 0.0) phi = PI_REF - phi;
    if (phi > PI_REF) phi = phi - 2.0 * PI_REF;
    if (phi < -PI_REF) phi = phi + 2.0 * PI_REF;
    if (!(phi < lo || phi > hi)) return;
    phi = (phi > hi) ? hi : ((phi < lo) ? lo : phi);
    V3<double> ax = n;
    const double al = O.length(ax);
    if (al != 0.0) ax = O.all(O.at(ax) / al);
    const double s = ::sin(phi / 2.0);
    const V3<double> as = O.all(O.at(ax) * s);
    const V3<double> m = O.rotate(qt<double>(as.x, as.y, as.z, ::cos(phi / 2.0)), n1);
    const V3<double> dq = O.own(O.all(O.cross(m, n2)));
    refresh(O, B);
    const double l = *lam;
    double len, dl = 0.0;
    V3<double> u;
    if (O.unit(dq, len, u)) {
        dl = ang_dlambda(O, B, h, 0.0, l, len, u);
        turn(O, B, O.row(B.I, O.all(-dl * O.at(u))));
    }
    __syncwarp(O.oct);
    if (O.lead()) *lam = l + dl;
}

// External constraints (pbd.cpp:81-379)
static __device__ void ext_solve(const WorldView<double>& W, const Oct& O, const ExtConstraint& C, double* lam, double h) {
    OctBody B = load_oct(W, O.side ? C.e2 : C.e1);
    const double* rl = O.side ? C.r2 : C.r1;
    const V3<double> r_lc = v3<double>(rl[0], rl[1], rl[2]);
    // one positional correction with lambda lam[k]
    auto positional = [&](int k, double compliance, V3<double> r, V3<double> dx) {
        refresh(O, B);
        const double l = lam[k];
        double len, dl = 0.0;
        V3<double> u;
        if (O.unit(dx, len, u)) {
            dl = pos_dlambda(O, B, r, h, compliance, l, len, u);
            pos_apply(O, B, r, dl, u);
        }
        __syncwarp(O.oct);
        if (O.lead()) lam[k] = l + dl;
    };
    auto angular = [&](int k, V3<double> dq) {
        refresh(O, B);
        const double l = lam[k];
        double len, dl = 0.0;
        V3<double> u;
        if (O.unit(dq, len, u)) {
            dl = ang_dlambda(O, B, h, C.compliance, l, len, u);
            turn(O, B, O.row(B.I, O.all(-dl * O.at(u))));
        }
        __syncwarp(O.oct);
        if (O.lead()) lam[k] = l + dl;
    };
    // an axis of the first and of the second body, in all lanes
    auto axes = [&](int k1, int k2, V3<double>& u1, V3<double>& u2) {
        const V3<double> mine = O.axis(B.q, O.side ? k2 : k1), theirs = O.other(mine);
        u1 = O.first(mine, theirs);
        u2 = O.second(mine, theirs);
    };
    // the anchors' separation
    auto apart = [&](V3<double> r) {
        const double p = O.at(B.x) + O.at(r);
        return O.all(p - O.other(p));
    };
    switch (C.type) {
    case CON_POSITIONAL: {  // pbd.cpp:81-97
        const V3<double> dist = O.own(v3<double>(C.distance[0], C.distance[1], C.distance[2]));
        const double x = O.at(B.x);
        const V3<double> dx = O.all((x - O.other(x)) - O.at(dist));
        positional(0, C.compliance, O.rotate(B.q, r_lc), dx);
    } break;
    case CON_MUTUAL_ORIENTATION: {  // pbd.cpp:156-173
        const Qt<double> oq = O.other(B.q);
        const Qt<double> aux = qmul(O.first(B.q, oq), qinverse(O.second(B.q, oq)));
        angular(0, O.own(v3<double>(2.0 * aux.x, 2.0 * aux.y, 2.0 * aux.z)));
    } break;
    case CON_HINGE: {  // pbd.cpp:245-299
        V3<double> u1, u2;
        axes(C.a1, C.a2, u1, u2);
        angular(1, O.own(O.all(O.cross(u1, u2))));
        const V3<double> r = O.rotate(B.q, r_lc);
        positional(0, 0.0, r, apart(r));
        if (C.limited) {
            V3<double> n1, n2;
            axes(C.l1, C.l2, n1, n2);
            axes(C.a1, C.a2, u1, u2);
            oct_limit(O, B, u1, n1, n2, C.lo, C.hi, h, lam + 2);
        }
    } break;
    case CON_SPHERICAL: {  // pbd.cpp:301-379
        const double EPS64 = 1e-50;
        const V3<double> r = O.rotate(B.q, r_lc);
        positional(0, 0.0, r, apart(r));
        V3<double> n1, n2;
        axes(C.a1, C.a2, n1, n2);
        V3<double> n = O.all(O.cross(n1, n2));
        double nl = O.length(n);
        if (nl > EPS64) oct_limit(O, B, O.all(O.at(n) / nl), n1, n2, C.lo, C.hi, h, lam + 1);
        V3<double> a1, a2, b1, b2;   // on the orientations after the swing correction
        axes(C.a1, C.a2, a1, a2);
        axes(C.l1, C.l2, b1, b2);
        n = O.all(O.at(a1) + O.at(a2));
        nl = O.length(n);
        if (nl > EPS64) {
            n = O.all(O.at(n) / nl);
            const double t1 = O.dot(O.at(n), O.at(b1)), t2 = O.dot(O.at(n), O.at(b2));
            n1 = O.all(O.at(b1) - t1 * O.at(n));
            n2 = O.all(O.at(b2) - t2 * O.at(n));
            const double l1 = O.length(n1), l2 = O.length(n2);
            if (l1 > EPS64 && l2 > EPS64) oct_limit(O, B, n, O.all(O.at(n1) / l1), O.all(O.at(n2) / l2), C.lo2, C.hi2, h, lam + 2);
        }
    } break;
    default: break;
    }
    store_oct(W, O, B);
}

// The contacts c[0, nc) of one pair on body `me` of this lane, position sweep. Contact record: r1_lc, lambda_n,
// r2_lc, lambda_t, normal, -.
__device__ inline void dsolve_pair(const WorldView<double>& W, const Oct& O, int me, double* c, int nc, double h) {
    const double mus_own = W.material[4 * me];
    const double mus = (mus_own + O.other(mus_own)) / 2.0;
    OctBody B = load_oct(W, me);
    const double4_32a px = W.prev_pos[me], pq = W.prev_rot[me];
    for (int i = 0; i < nc; ++i, c += 12) {
        double ln = c[3], lt = c[7];
        const bool acts = oct_contact(O, B, v3<double>(c[4 * O.side], c[4 * O.side + 1], c[4 * O.side + 2]),
                                      O.own(v3<double>(c[8], c[9], c[10])), mus, v3<double>(px.x, px.y, px.z),
                                      qt<double>(pq.x, pq.y, pq.z, pq.w), h, ln, lt);
        if (!acts) continue;
        // all lanes hold the same multipliers: a lane of each body writes one
        __syncwarp(O.oct);
        if (O.c == 0) c[O.side ? 7 : 3] = O.side ? lt : ln;
    }
    store_oct(W, O, B);
}

// and velocity sweep (pbd.cpp:646-711)
__device__ inline void dvsolve_pair(const WorldView<double>& W, const Oct& O, int me, const double* c, int nc, double h) {
    // anchors rotated by the current orientation (the poses do not change here)
    const double4_32a q4 = W.rot[me];
    const Qt<double> q = qt<double>(q4.x, q4.y, q4.z, q4.w);
    double sI[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) sI[i] = W.inv_inertia[6 * me + i];
    const V3<double> I = O.tensor(q, sI);
    const double invm = W.inv_mass[me];
    const bool fixed = W.fixed[me] != 0;
    V3<double> vel = v3<double>(W.vel[3 * me], W.vel[3 * me + 1], W.vel[3 * me + 2]);
    V3<double> om = v3<double>(W.omega[3 * me], W.omega[3 * me + 1], W.omega[3 * me + 2]);
    const V3<double> pv = v3<double>(W.prev_vel[3 * me], W.prev_vel[3 * me + 1], W.prev_vel[3 * me + 2]);
    const V3<double> pw = v3<double>(W.prev_omega[3 * me], W.prev_omega[3 * me + 1], W.prev_omega[3 * me + 2]);
    const double mud_own = W.material[4 * me + 1], e_own = W.material[4 * me + 2];
    const double mud = (mud_own + O.other(mud_own)) / (double)2.0f;
    const double e = e_own * O.other(e_own);
    const int mine = 4 * O.side + O.c;   // lambda_n / h of eight contacts at once
    double fns = 0.0;
    for (int i = 0; i < nc; ++i) {
        if ((i & 7) == 0) fns = (i + mine < nc ? c[12 * (i + mine) + 3] : 0.0) / h;
        const double fn = __shfl_sync(O.oct, fns, i & 7, 8);
        const double* ci = c + 12 * i;
        const V3<double> r = O.rotate(q, v3<double>(ci[4 * O.side], ci[4 * O.side + 1], ci[4 * O.side + 2]));
        const V3<double> n = O.own(v3<double>(ci[8], ci[9], ci[10]));
        const double nc_ = O.at(n);
        const double u = O.at(vel) + O.cross(om, r);
        const double v = u - O.other(u);
        const double vn = O.dot(nc_, v);
        const double vt = v - vn * nc_;
        const V3<double> t = O.all(vt), ts = O.all(vt * vt);
        const double x1 = mud * ::fabs(fn), x2 = ::sqrt(ts.x + ts.y + ts.z);
        double fact = (x1 < x2) ? x1 : x2;
        const double tn = (t.x != 0.0 || t.y != 0.0 || t.z != 0.0) ? O.at(t) / x2 : 0.0;
        double dv = 0.0 + -fact * tn;
        const double ut = O.at(pv) + O.cross(pw, r);
        const double vntil = O.dot(nc_, ut - O.other(ut));
        const double m = -e * vntil;
        fact = -vn + ((m < 0.0) ? m : 0.0);
        dv = dv + fact * nc_;
        const double a = O.cross(r, n);
        const double w = invm + O.dot(a, O.row(I, O.all(a)));
        const double P = (1.0 / (w + O.other(w))) * dv;
        const double dw = O.row(I, O.all(O.cross(r, O.all(P))));
        if (!fixed) {
            vel = O.all(O.at(vel) + invm * P);
            om = O.all(O.at(om) + dw);
        }
    }
    if (!fixed && O.c == 0) {
        W.vel[3 * me] = vel.x; W.vel[3 * me + 1] = vel.y; W.vel[3 * me + 2] = vel.z;
        W.omega[3 * me] = om.x; W.omega[3 * me + 1] = om.y; W.omega[3 * me + 2] = om.z;
    }
}

// Predict (pbd.cpp:537-577) of body b by its four lanes, and the FP32 copy of the pose
__device__ __forceinline__ void oct_predict(const WorldView<double>& W, const Oct& O, int b, double h) {
    const double4_32a p4 = W.pos[b], q4 = W.rot[b];
    V3<double> x = v3<double>(p4.x, p4.y, p4.z);
    Qt<double> q = qt<double>(q4.x, q4.y, q4.z, q4.w);
    if (!W.fixed[b] && W.active[b]) {
        double L[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) L[i] = W.inv_inertia[6 * b + i];
        const Oct::Rot R = O.matrix(q);
        const V3<double> Iinv = O.tensor(R, L);
#pragma unroll
        for (int i = 0; i < 6; ++i) L[i] = W.inertia[6 * b + i];
        const V3<double> I = O.tensor(R, L);
        const int c = O.c < 3 ? O.c : 2;
        const V3<double> w = v3<double>(W.omega[3 * b], W.omega[3 * b + 1], W.omega[3 * b + 2]);
        const double v = W.vel[3 * b + c] + h * W.inv_mass[b] * W.force[3 * b + c];
        const V3<double> Iw = O.all(O.row(I, w));
        const V3<double> g = O.all(W.torque[3 * b + c] - O.cross(w, Iw));
        const double wc = O.at(w) + h * O.row(Iinv, g);
        const V3<double> wn = O.all(wc);
        x = O.all(O.at(x) + h * v);
        q = O.normalize(O.at4(q) + h * 0.5 * O.mul(qt<double>(wn.x, wn.y, wn.z, 0.0), q));
        __syncwarp(O.quad);   // the old velocities are read
        if (O.c < 3) {
            W.vel[3 * b + c] = v;
            W.omega[3 * b + c] = wc;
        }
    }
    if (O.c != 0) return;
    W.prev_pos[b] = p4;
    W.prev_rot[b] = q4;
    W.pos[b] = make_double4_32a(x.x, x.y, x.z, 0.0);
    W.rot[b] = make_double4_32a(q.x, q.y, q.z, q.w);
    W.pose_f[2 * b] = make_float4((float)x.x, (float)x.y, (float)x.z, 0.f);
    W.pose_f[2 * b + 1] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
}

// PBD velocity update (pbd.cpp:623-643) of body b by its four lanes; inv_h = 1 / h
__device__ __forceinline__ void oct_velocity(const WorldView<double>& W, const Oct& O, int b, double inv_h) {
    if (W.fixed[b] || !W.active[b]) return;
    const double4_32a p = W.pos[b], q = W.rot[b], pp = W.prev_pos[b], pq = W.prev_rot[b];
    const double dq = O.mul(qt<double>(q.x, q.y, q.z, q.w), qinverse(qt<double>(pq.x, pq.y, pq.z, pq.w)));
    const bool ahead = __shfl_sync(O.quad, dq, 3, 4) >= 0.0;
    if (O.c == 3) return;
    const int i = 3 * b + O.c;
    W.prev_vel[i] = W.vel[i];
    W.prev_omega[i] = W.omega[i];
    W.vel[i] = inv_h * (O.at(p) - O.at(pp));
    const double two = 2.0 * inv_h;   // the reference's 2 / h: the same double
    W.omega[i] = (ahead ? two : -two) * dq;
}

}  // namespace rp
