// The narrowphase of two single hulls of at most 64 vertices by one warp: the common pair of the phase-major
// kernels. (rp_narrow.cuh holds the same algorithms for any collider.)
//
// Support mapping runs on registers: lane i holds vertices i and i + 32 of both hulls, so a support call is two
// dot products a lane, a warp reduction and a shuffle, without a load. Topology comes in byte records (RecTables
// in rp_world.h), loaded four bytes a lane: a vertex record (its faces and neighbours) and a face record (its
// loop, its neighbour faces and the first vertex of each). The general code walks the same
// lists through five dependent table loads (about 600 cycles each when they miss L1); a pair's contact
// manifold waited for about twenty of them and now waits for four.
#pragma once
#include "rp_step.cuh"

namespace rp {

// Lane i's vertices i and i + 32 of a hull, in the pair frame
template <typename R>
struct RegHull {
    V3<R> v0, v1;
    int nv;
};

template <typename R>
__device__ __forceinline__ RegHull<R> load_reghull(const WorldView<R>& W, const HullRef& h, V3<R> off) {
    RegHull<R> H;
    const int lane = (int)lane_id();
    const V3<R>* tv = (const V3<R>*)(W.tverts) + h.tv_off;
    H.nv = h.nv;
    H.v0 = H.v1 = v3<R>(0, 0, 0);
    if (lane < h.nv) H.v0 = vadd(tv[lane], off);
    if (lane + 32 < h.nv) H.v1 = vadd(tv[lane + 32], off);
    return H;
}

// vertex idx (the same in every lane)
template <typename R>
__device__ __forceinline__ V3<R> reg_vertex(const RegHull<R>& H, int idx) {
    const V3<R> v = idx >= 32 ? H.v1 : H.v0;
    const int src = idx & 31;
    return v3<R>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src), __shfl_sync(0xffffffffu, v.z, src));
}

// each lane's first best vertex along d (support.cpp:5-14: strict >, the first maximum wins)
template <typename R>
__device__ __forceinline__ void reg_best(const RegHull<R>& H, V3<R> d, R& best, int& bi) {
    const int lane = (int)lane_id();
    best = sizeof(R) == 4 ? (R)-FLT_MAX : (R)-DBL_MAX;
    bi = 0x7fffffff;
    if (lane < H.nv) {
        const R dot = vdot(H.v0, d);
        if (dot > best) { best = dot; bi = lane; }
    }
    if (lane + 32 < H.nv) {
        const R dot = vdot(H.v1, d);
        if (dot > best) { best = dot; bi = lane + 32; }
    }
}

// the support vertices of a along d and of b along nd
template <typename R>
__device__ __forceinline__ void reg_support2(const RegHull<R>& a, const RegHull<R>& b, V3<R> d, V3<R> nd, int& ia, int& ib) {
    R ba, bb;
    reg_best(a, d, ba, ia);
    reg_best(b, nd, bb, ib);
    if constexpr (sizeof(R) == 4) {
        warp_argmax_first(ba, ia);
        warp_argmax_first(bb, ib);
    } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            R ova = __shfl_xor_sync(0xffffffffu, ba, o), ovb = __shfl_xor_sync(0xffffffffu, bb, o);
            int oia = __shfl_xor_sync(0xffffffffu, ia, o), oib = __shfl_xor_sync(0xffffffffu, ib, o);
            if (ova > ba || (ova == ba && oia < ia)) { ba = ova; ia = oia; }
            if (ovb > bb || (ovb == bb && oib < ib)) { bb = ovb; ib = oib; }
        }
    }
    if (ia == 0x7fffffff) ia = 0;
    if (ib == 0x7fffffff) ib = 0;
}

// support_point_of_minkowski_difference (support.cpp:29-39) on registers, the form gjk_run and epa take
template <typename R>
struct RegMink {
    const RegHull<R>& a;
    const RegHull<R>& b;
    __device__ __forceinline__ V3<R> operator()(V3<R> d) const {
        int ia, ib;
        reg_support2(a, b, d, vscale((R)-1.0, d), ia, ib);
        return vsub(reg_vertex(a, ia), reg_vertex(b, ib));
    }
};

// A topology record whose first 128 bytes the warp holds, four bytes a lane; longer ones (a hub of more than
// 40 edges or so) are read from memory beyond that.
struct Rec {
    const unsigned char* p;
    unsigned w;
    __device__ __forceinline__ Rec(const unsigned char* base, int line, int index, int stride)
        : p(base + 128 * ((size_t)line + (size_t)index * stride)), w(reinterpret_cast<const unsigned*>(p)[lane_id()]) {}
    // byte i; every lane calls it together
    __device__ __forceinline__ int operator[](int i) const {
        int v = (int)((__shfl_sync(0xffffffffu, w, (i >> 2) & 31) >> (8 * (i & 3))) & 255u);
        if (i >= 128) v = p[i];
        return v;
    }
};

// One Sutherland-Hodgman pass (sh_pass, without its all-inside shortcut): a lane per polygon edge, the output
// places from two ballots. Returns the output count.
template <typename R, bool REMOVE_ONLY>
__device__ __forceinline__ int clip_pass(const V3<R>* in, int n, V3<R>* out, V3<R> pn, V3<R> pp, int& status) {
    const unsigned lane = lane_id(), below = (1u << lane) - 1u;
    int carry = 0;
    for (int base = 0; base < n; base += WARP) {
        const int j = base + (int)lane;
        bool first = false, second = false;   // the edge emits its crossing (or end point), then its end point
        V3<R> o0 = v3<R>(0, 0, 0), end = v3<R>(0, 0, 0);
        if (j < n) {
            end = in[j];
            const bool ei = in_plane(pn, pp, end);
            o0 = end;
            first = ei;
            if (!REMOVE_ONLY) {
                const V3<R> start = in[j == 0 ? n - 1 : j - 1];
                const bool si = in_plane(pn, pp, start);
                V3<R> t;
                if (si != ei && plane_edge(pn, pp, start, end, t)) {
                    o0 = t;
                    first = true;
                    second = ei;
                }
            }
        }
        const unsigned m1 = __ballot_sync(0xffffffffu, first), m2 = REMOVE_ONLY ? 0u : __ballot_sync(0xffffffffu, second);
        const int pos = carry + __popc(m1 & below) + __popc(m2 & below);
        if (first) { if (pos < CLIP_MAX) out[pos] = o0; else status |= ST_CLIP_OVERFLOW; }
        if (second) { if (pos + 1 < CLIP_MAX) out[pos + 1] = end; else status |= ST_CLIP_OVERFLOW; }
        carry += __popc(m1) + __popc(m2);
    }
    __syncwarp();
    return carry < CLIP_MAX ? carry : CLIP_MAX;
}

// convex_convex_contact_manifold (clipping.cpp:249-341) of two register hulls; sm.va / sm.vb hold the staged
// vertices (pair frame) for the per-lane lookups.
template <typename R, bool EXACT>
__device__ void hull_manifold(NarrowSmem<R>& sm, const WorldView<R>& W, const RegHull<R>& ra, const RegHull<R>& rb, const HullRef& ha,
                              const HullRef& hb, int body_a, int body_b, V3<R> normal, V3<double> normal64, const PairFrame<R, EXACT>& fr) {
    const int lane = (int)lane_id();
    const V3<R> inv_n = vinv(normal);
    int s1, s2;
    reg_support2(ra, rb, normal, inv_n, s1, s2);
    const unsigned char* topo = W.topo_rec;
    const Rec w1(topo, ha.vrec, s1, ha.vstride), w2(topo, hb.vrec, s2, hb.vstride);
    const V3<R>* na = (const V3<R>*)(W.tnorms) + ha.tn_off;
    const V3<R>* nb = (const V3<R>*)(W.tnorms) + hb.tn_off;
    const int nf1 = w1[0], nn1 = w1[1], nf2 = w2[0], nn2 = w2[1];
    // get_face_with_most_fitting_normal over vertex -> faces (first max wins)
    R best1 = sizeof(R) == 4 ? -FLT_MAX : -(R)DBL_MAX, best2 = best1;
    int k1 = 0x7fffffff, k2 = 0x7fffffff;
    for (int base = 0; base < max(nf1, nf2); base += WARP) {
        const int k = base + lane;
        const int fa = w1[2 + k], fb = w2[2 + k];
        if (k < nf1) {
            const R p = vdot(na[fa], normal);
            if (p > best1) { best1 = p; k1 = k; }
        }
        if (k < nf2) {
            const R p = vdot(nb[fb], inv_n);
            if (p > best2) { best2 = p; k2 = k; }
        }
    }
    warp_argmax_first(best1, k1);
    warp_argmax_first(best2, k2);
    const int f1 = w1[2 + (k1 == 0x7fffffff ? 0 : k1)], f2 = w2[2 + (k2 == 0x7fffffff ? 0 : k2)];
    // both faces' records and normals, before it is known which is the reference
    const Rec r1(topo, ha.frec, f1, ha.fstride), r2(topo, hb.frec, f2, hb.fstride);
    const V3<R> n1 = na[f1], n2 = nb[f2];
    // get_edge_with_most_fitting_normal: candidates in (i, j, normal / inverted) order
    const V3<R> sp1 = reg_vertex(ra, s1), sp2 = reg_vertex(rb, s2);
    R bestE = sizeof(R) == 4 ? -FLT_MAX : -(R)DBL_MAX;
    int bestK = 0x7fffffff;
    for (int base = 0; base < nn1 * nn2; base += WARP) {
        const int k = base + lane;
        const int i = k / nn2, j = k - i * nn2;
        const int va = w1[2 + nf1 + i], vb = w2[2 + nf2 + j];
        if (k < nn1 * nn2) {
            V3<R> e1 = vsub(sp1, sm.va[va]);
            V3<R> e2 = vsub(sp2, sm.vb[vb]);
            V3<R> cn = vnorm(vcross(e1, e2));
            V3<R> ci = vinv(cn);
            R d0 = vdot(cn, normal);
            if (d0 > bestE) { bestE = d0; bestK = 2 * k; }
            R d1 = vdot(ci, normal);
            if (d1 > bestE) { bestE = d1; bestK = 2 * k + 1; }
        }
    }
    warp_argmax_first(bestE, bestK);
    const bool edges = bestK != 0x7fffffff;
    const R d1 = vdot(n1, normal), d2 = vdot(n2, inv_n), de = edges ? bestE : (R)0;
    if (de > d1 + (R)0.0001 && de > d2 + (R)0.0001) {
        // collision_distance_between_skew_lines (clipping.cpp:210-239)
        const int k = edges ? bestK >> 1 : 0;
        const V3<R> q1 = sm.va[w1[2 + nf1 + (edges ? k / nn2 : 0)]], q2 = sm.vb[w2[2 + nf2 + (edges ? k % nn2 : 0)]];
        V3<R> l1, l2;
        const bool ok = skew_points(sp1, vsub(edges ? q1 : sm.va[0], sp1), sp2, vsub(edges ? q2 : sm.vb[0], sp2), l1, l2);
        if (!ok && lane == 0) atomicOr(&sm.status, (int)(ST_DEGENERATE | ST_DEG_SKEW));
        push_contact(sm, fr, l1, l2, normal, ok && lane == 0);
        return;
    }
    bool ref1 = d1 > d2;
    // screen in FP32: |d1 - d2| below 1e-5 (within the float subtraction's rounding: 1.1e-5 covers it)
    if (!EXACT && fabsf((float)d1 - (float)d2) < 1.1e-5f) {
        // Nearly parallel faces: the reference decides d1 > d2 in FP64, below FP32 resolution of the dot products.
        // For unit vectors 1 - <m, n> = |m - n|^2 / 2, which FP32 resolves far better near zero: with each
        // vector within e of its FP64 value, |m - n|^2 is within 2 e |m - n| + e^2. e = 2e-6 covers the FP32
        // normals (about 5e-7 off). The FP64 comparison (7500 cycles of one lane, 30 % of this kernel before)
        // is left for faces parallel to within about 1e-5 rad, one face a lane.
        const V3<R> u1 = vsub(n1, normal), u2 = vadd(n2, normal);
        const R q1 = vdot(u1, u1), q2 = vdot(u2, u2), e = (R)2e-6;
        if (fabsf((float)(q1 - q2)) > (float)((R)2 * e * (sqrtf((float)q1) + sqrtf((float)q2)) + (R)4 * e * e)) {
            ref1 = q1 < q2;
        } else {
            double d = 0.0;
            if (lane < 2) {
                const double4_32a q = W.rot[lane ? body_b : body_a];
                const V3<double> n = lane ? vinv(normal64) : normal64;
                d = turned_dot(W.face_normal + 3 * (lane ? hb.face_off + f2 : ha.face_off + f1), q.x, q.y, q.z, q.w, n.x, n.y, n.z);
            }
            ref1 = __shfl_sync(0xffffffffu, d, 0) > __shfl_sync(0xffffffffu, d, 1);
        }
    }
    // incident polygon and boundary planes (build_boundary_planes, clipping.cpp:121-134)
    const Rec rr = ref1 ? r1 : r2, ri = ref1 ? r2 : r1;
    const V3<R>* rn = ref1 ? na : nb;
    const V3<R>* rv = ref1 ? sm.va : sm.vb;
    const V3<R>* iv = ref1 ? sm.vb : sm.va;
    const int nref = rr[0], neighbours = rr[1], corners = ri[0];
    // a face has as many neighbours as faces share a vertex with it, up to the record's 255
    if ((neighbours > CLIP_MAX || corners > CLIP_MAX) && lane == 0) atomicOr(&sm.status, (int)ST_CLIP_OVERFLOW);
    const int npl = min(neighbours, CLIP_MAX), ninc = min(corners, CLIP_MAX);
    for (int base = 0; base < ninc; base += WARP) {
        const int k = base + lane, v = ri[2 + k];
        if (k < ninc) sm.u.clip.buf[0][k] = iv[v];
    }
    for (int base = 0; base < npl; base += WARP) {
        const int k = base + lane, nf = rr[2 + nref + k], v = rr[2 + nref + neighbours + k];
        if (k < npl) {
            sm.u.clip.pp[k] = rv[v];
            sm.u.clip.pn[k] = vinv(rn[nf]);
        }
    }
    __syncwarp();
    int st = 0;
    int n = ninc, cur = 0;
    // Planes in order; one with every vertex inside leaves the polygon as it is, so 32 planes are tested at a
    // time, a plane a lane, and only the first with a vertex outside is clipped against before the rest are
    // tested again.
    for (int base = 0; base < npl && n > 0; base += WARP) {
        const int k = base + lane;
        unsigned todo = npl - base >= 32 ? 0xffffffffu : (1u << (npl - base)) - 1u;
        while (todo && n > 0) {
            bool out = false;
            if (k < npl) {
                const V3<R> pn = sm.u.clip.pn[k], pp = sm.u.clip.pp[k];
                for (int j = 0; j < n; ++j) out |= !in_plane(pn, pp, sm.u.clip.buf[cur][j]);
            }
            todo &= __ballot_sync(0xffffffffu, out);
            if (!todo) break;
            const int p = base + __ffs(todo) - 1;
            n = clip_pass<R, false>(sm.u.clip.buf[cur], n, sm.u.clip.buf[cur ^ 1], sm.u.clip.pn[p], sm.u.clip.pp[p], st);
            cur ^= 1;
            // the planes after p see the new polygon
            todo = (npl - base >= 32 ? 0xffffffffu : (1u << (npl - base)) - 1u) & ~((2u << (p - base)) - 1u);
        }
    }
    const V3<R> ref_n = vinv(ref1 ? n1 : n2);
    const V3<R> ref_p = rv[rr[2]];
    if (n > 0) {
        n = clip_pass<R, true>(sm.u.clip.buf[cur], n, sm.u.clip.buf[cur ^ 1], ref_n, ref_p, st);
        cur ^= 1;
    }
    if (st && lane == 0) atomicOr(&sm.status, (int)st);
    clipped_contacts<R, EXACT>(sm, fr, sm.u.clip.buf[cur], n, ref1, ref_n, ref_p, normal);
}

}  // namespace rp
