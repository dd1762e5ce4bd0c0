// Adjoint kernels of the substep (rp_adjoint.cuh, rp_adjoint_contact.cuh) and their launcher.
// Built without FMA contraction: the scalar forward pass then reproduces the all-FP64 step.
#include "rp_adjoint_contact.cuh"

namespace rp {

// Body state at a substep boundary: x[3], q[4], v[3], w[3]
constexpr int ADJ_STATE = 13;
// Tape leaves per body: the 13 state values, the inverse mass, static and dynamic friction
constexpr int ADJ_LEAVES = 16;
// Checkpoint per body: the state, the deactivation time and the awake flag
constexpr int ADJ_CKPT = 15;
constexpr int ADJ_WARPS = 16;          // warps of a scalar-pass block: pairs whose narrowphase runs at once
constexpr int TAPE_BLOCK = 128;
constexpr int REV_BLOCK = 256;
// shared memory of the reverse sweep: the adjoints of the last entries, and a chunk's edges and entries
constexpr int ADJ_RING = 8192, CHUNK_EDGES = 4096, CHUNK_ENTRIES = 2048;

// The body's inertia tensors at its exact FP64 values, as functions of its inverse mass: the default
// inertia is a point-mass sum (colliders_get_default_inertia_tensor, collider.cpp:448-494), so
// I = m I_unit and I^-1 = invm I_unit^-1, with d I^-1 / d invm = I^-1 / invm, d I / d invm = -I / invm.
template <typename S>
__device__ void g_inertia(GBody<S>& B, const AdjointScene& sc, int i, double invm) {
    S si[6], sI[6];
    for (int k = 0; k < 6; ++k) {
        const double vi = sc.inv_inertia[6 * i + k], vI = sc.inertia[6 * i + k];
        if constexpr (sizeof(S) == sizeof(double)) {
            si[k] = vi;
            sI[k] = vI;
        } else {
            si[k] = a_op1(vi, B.invm, vi / invm);
            sI[k] = a_op1(vI, B.invm, -vI / invm);
        }
    }
    B.Iinv = msym(si);
    B.I = msym(sI);
}

template <typename S>
__device__ __forceinline__ S g_input(double x) {
    if constexpr (sizeof(S) == sizeof(double)) return x;
    else return a_leaf(x);
}

// Body i at the start of a substep. With S = AVar its 16 inputs become tape leaves: 13 state values, inverse
// mass, static and dynamic friction (called for all bodies in order first, so ids 16 i .. 16 i + 15).
template <typename S>
__device__ void g_body(GBody<S>& b, const double* start, const AdjointScene& sc, int i, const uint8_t* active) {
    const double* st = start + ADJ_STATE * i;
    S vals[ADJ_LEAVES];
    for (int k = 0; k < ADJ_STATE; ++k) vals[k] = g_input<S>(st[k]);
    vals[13] = g_input<S>(sc.invm[i]);
    vals[14] = g_input<S>(sc.material[3 * i]);
    vals[15] = g_input<S>(sc.material[3 * i + 1]);
    b.x = v3<S>(vals[0], vals[1], vals[2]);
    b.q = qt<S>(vals[3], vals[4], vals[5], vals[6]);
    b.v = v3<S>(vals[7], vals[8], vals[9]);
    b.w = v3<S>(vals[10], vals[11], vals[12]);
    b.invm = vals[13];
    b.mus = vals[14];
    b.mud = vals[15];
    b.rest = S(sc.material[3 * i + 2]);
    const double* pv = sc.prev_vel + 6 * i;
    b.pv = v3<S>(S(pv[0]), S(pv[1]), S(pv[2]));
    b.pw = v3<S>(S(pv[3]), S(pv[4]), S(pv[5]));
    b.fixed = sc.fixed[i] != 0;
    b.active = active[i] != 0;
}
template <typename S>
__device__ void g_fall(GBody<S>& b, const AdjointScene& sc, int i, const AdjointParams& P, double h) {
    if (!b.fixed) {
        g_inertia(b, sc, i, sc.invm[i]);
    } else {
        // a fixed body's tensors are zero (entity_create_fixed): constants, as its inverse mass
        const S z[6] = {S(0.0), S(0.0), S(0.0), S(0.0), S(0.0), S(0.0)};
        b.Iinv = msym(z);
        b.I = msym(z);
    }
    // gravity as the caller's force -g m (stack.cpp:93-96), formed as the host forms it
    const S Fy = b.fixed ? S(0.0) : S(-P.gravity * 1.0) / b.invm;
    g_predict(b, v3<S>(S(0.0), Fy, S(0.0)), h);
}
// pairs whose bodies are both fixed or asleep are skipped (pbd.cpp:590-593)
__device__ __forceinline__ bool g_skip(const AdjointScene& sc, const uint8_t* active, int2 p) {
    return (sc.fixed[p.x] || !active[p.x]) && (sc.fixed[p.y] || !active[p.y]);
}
template <typename S>
__device__ __forceinline__ void g_node(const AdjointScene& sc, GBody<S>* B, GCon<S>* con, S* lam, int node, double h) {
    if (node < sc.ne) {
        const ExtConstraint& C = sc.ext[node];
        g_ext_solve(B[C.e1 - sc.body0], B[C.e2 - sc.body0], C, lam + 4 * node, h);
    } else {
        GCon<S>& c = con[node - sc.ne];
        g_collision_solve(B[c.a], B[c.b], c, h);
    }
}

// A block's scalar scratch of one scene
struct Forward {
    GBody<double>* B;
    GScene<double> X;          // contacts of the scene
    GCon<double>* stage;       // [ADJ_WARPS CMAX] contacts of a round of pairs
    GClip<double>* clip;       // [ADJ_WARPS]
    GEpa* epa;                 // [ADJ_WARPS]
};

__device__ Forward g_forward_view(const AdjointScene& sc) {
    Forward F;
    F.B = reinterpret_cast<GBody<double>*>(sc.bodies_d);
    F.X.tv = F.X.tvv = reinterpret_cast<V3<double>*>(sc.tv_d);   // the scalar pass's values are the geometry itself
    F.X.tn = F.X.tnv = reinterpret_cast<V3<double>*>(sc.tn_d);
    F.X.con = reinterpret_cast<GCon<double>*>(sc.con_d);
    F.X.ncon = 0;
    F.X.con_cap = sc.contact_cap;
    F.stage = reinterpret_cast<GCon<double>*>(sc.stage_d);
    F.clip = reinterpret_cast<GClip<double>*>(sc.clip_d);
    F.epa = reinterpret_cast<GEpa*>(sc.epa);
    F.X.clip = F.clip;
    F.X.epa = F.epa;
    return F;
}

__shared__ int s_cnt[ADJ_WARPS + 1];
__shared__ int s_np, s_lev, s_ncon;

// The scalar substep by a whole block. Bodies, hull vertices and the nodes of one level of the solves are
// independent and go to different threads; each pair's serial GJK, EPA and clipping runs on its own warp,
// whose lanes would only diverge. The contacts keep the pairs' order, and a level of the solves holds nodes
// with no movable body in common whose predecessors are in earlier levels, so every value is the serial
// substep's. FP64 issue bounds it (a 64th of the FP32 rate, whatever the lanes): 20 substeps of 24 rows of
// 12 dominoes took one thread a scene 97 ms and take a block 15 ms.
__device__ void g_substep_block(Forward& F, const double* start, double* out, const AdjointScene& sc, const AdjointParams& P,
                                const int2* pairs, int np, const uint8_t* active) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nb = sc.nb;
    const double h = P.dt / P.substeps;
    GBody<double>* B = F.B;
    for (int i = tid; i < nb; i += nt) {
        g_body(B[i], start, sc, i, active);
        g_fall(B[i], sc, i, P, h);
        sc.stamp[i] = 0;
    }
    int ncon = 0;
    if (P.collisions) {
        __syncthreads();
        for (int k = tid; k < np; k += nt) {
            if (g_skip(sc, active, pairs[k])) continue;
            sc.stamp[pairs[k].x] = 1;
            sc.stamp[pairs[k].y] = 1;
        }
        __syncthreads();
        for (int i = warp; i < nb; i += ADJ_WARPS)
            if (sc.stamp[i]) g_transform(sc, P.geom, B[i], i, F.X, lane, 32);
        __syncthreads();
        for (int k0 = 0; k0 < np; k0 += ADJ_WARPS) {
            const int k = k0 + warp;
            if (lane == 0) {
                GScene<double> X = F.X;
                X.con = F.stage + warp * CMAX;
                X.con_cap = CMAX;
                X.clip = F.clip + warp;
                X.epa = F.epa + warp;
                if (k < np && !g_skip(sc, active, pairs[k])) g_pair_contacts(sc, P.geom, X, B, pairs[k].x, pairs[k].y);
                s_cnt[warp] = X.ncon;
            }
            __syncthreads();
            int at = ncon, total = ncon;
            for (int w = 0; w < ADJ_WARPS; ++w) {
                if (w == warp) at = total;
                total += s_cnt[w];
            }
            for (int c = lane; c < s_cnt[warp]; c += 32)
                if (at + c < sc.contact_cap) F.X.con[at + c] = F.stage[warp * CMAX + c];
            if (total > sc.contact_cap && tid == 0) atomicOr(sc.status, ADJ_ST_CONTACTS);
            ncon = min(total, sc.contact_cap);
            __syncthreads();
        }
    }
    // levels of the nodes: joints, then contacts, in their serial order
    const int nodes = sc.ne + ncon;
    __syncthreads();
    if (tid == 0) {
        int top = 0;
        for (int i = 0; i < nb; ++i) sc.stamp[i] = 0;
        for (int k = 0; k < nodes; ++k) {
            const int a = k < sc.ne ? sc.ext[k].e1 - sc.body0 : F.X.con[k - sc.ne].a;
            const int c = k < sc.ne ? sc.ext[k].e2 - sc.body0 : F.X.con[k - sc.ne].b;
            const int l = max(sc.fixed[a] ? 0 : sc.stamp[a], sc.fixed[c] ? 0 : sc.stamp[c]) + 1;
            sc.stamp[a] = l;
            sc.stamp[c] = l;
            sc.node_level[k] = l;
            top = max(top, l);
        }
        s_lev = top;
    }
    for (int e = tid; e < 4 * sc.ne; e += nt) sc.lam_d[e] = 0.0;
    __syncthreads();
    const int levels = s_lev;
    for (int it = 0; it < P.pos_iters; ++it)
        for (int l = 1; l <= levels; ++l) {
            for (int k = tid; k < nodes; k += nt)
                if (sc.node_level[k] == l) g_node(sc, B, F.X.con, sc.lam_d, k, h);
            __syncthreads();
        }
    for (int i = tid; i < nb; i += nt) g_velocity(B[i], h);
    __syncthreads();
    if (ncon > 0)
        for (int l = 1; l <= levels; ++l) {
            for (int k = sc.ne + tid; k < nodes; k += nt)
                if (sc.node_level[k] == l) g_contact_velocity(B[F.X.con[k - sc.ne].a], B[F.X.con[k - sc.ne].b], F.X.con[k - sc.ne], h);
            __syncthreads();
        }
    for (int i = tid; i < nb; i += nt) {
        double* o = out + ADJ_STATE * i;
        o[0] = B[i].x.x; o[1] = B[i].x.y; o[2] = B[i].x.z;
        o[3] = B[i].q.x; o[4] = B[i].q.y; o[5] = B[i].q.z; o[6] = B[i].q.w;
        o[7] = B[i].v.x; o[8] = B[i].v.y; o[9] = B[i].v.z;
        o[10] = B[i].w.x; o[11] = B[i].w.y; o[12] = B[i].w.z;
    }
    __syncthreads();
}

// Scalar trajectory, a block per scene. seg < 0: all frames from the start, with a checkpoint at every K-th
// frame start, the loss and its seed. Else: segment seg again from its checkpoint. Either way every substep's
// start state and every frame's pairs and awake flags go to the segment's slots, so that after the forward
// pass they are the last segment's.
__global__ void __launch_bounds__(32 * ADJ_WARPS) k_adjoint_forward(const AdjointScene* scenes, AdjointParams P, int seg) {
    const AdjointScene& sc = scenes[blockIdx.x];
    const int tid = threadIdx.x, nt = blockDim.x;
    const long long t0 = clock64();
    const int nb = sc.nb, S_ = P.substeps, K = P.checkpoint_every;
    const size_t stride = (size_t)ADJ_STATE * nb, cstride = (size_t)ADJ_CKPT * nb;
    Forward F = g_forward_view(sc);
    if (tid == 0 && seg < 0) sc.status[0] = 0;
    const int f0 = seg < 0 ? 0 : seg * K, f1 = seg < 0 ? P.frames : min(P.frames, f0 + K);
    if (seg < 0) {
        for (size_t k = tid; k < stride; k += nt) sc.segment[k] = sc.start[k];
        for (int i = tid; i < nb; i += nt) { sc.deact[i] = sc.deact0[i]; sc.active[i] = sc.active0[i]; }
    } else {
        const double* ck = sc.checkpoints + (size_t)seg * cstride;
        for (size_t k = tid; k < stride; k += nt) sc.segment[k] = ck[k];
        for (int i = tid; i < nb; i += nt) { sc.deact[i] = ck[stride + i]; sc.active[i] = ck[stride + nb + i] != 0.0 ? 1 : 0; }
    }
    __syncthreads();
    double* cur = sc.segment;
    for (int f = f0; f < f1; ++f) {
        const int fl = f % K;
        if (fl == 0) {
            // the state at a segment's start moves to its first slot (the last substep of a segment ends one past it)
            if (cur != sc.segment) {
                for (size_t k = tid; k < stride; k += nt) sc.segment[k] = cur[k];
                cur = sc.segment;
                __syncthreads();
            }
            if (seg < 0) {
                double* ck = sc.checkpoints + (size_t)(f / K) * cstride;
                for (size_t k = tid; k < stride; k += nt) ck[k] = cur[k];
                for (int i = tid; i < nb; i += nt) { ck[stride + i] = sc.deact[i]; ck[stride + nb + i] = sc.active[i]; }
            }
        }
        int2* fp = sc.pairs + (size_t)fl * sc.pair_cap;
        uint8_t* fa = sc.active_seg + (size_t)fl * nb;
        __syncthreads();
        if (tid < 32) {
            const int np = g_broad(sc, P.geom, cur, fp);
            __syncwarp();
            if (tid == 0) {
                g_islands(sc, cur, fp, np, P.dt);
                for (int i = 0; i < nb; ++i) fa[i] = sc.active[i];
                sc.npairs[fl] = np;
                s_np = np;
            }
        }
        __syncthreads();
        const int np = s_np;
        for (int u = 0; u < S_; ++u) {
            g_substep_block(F, cur, cur + stride, sc, P, fp, np, fa);
            cur += stride;
        }
    }
    if (tid != 0) return;
    if (seg >= 0) {
        sc.prof[1] += clock64() - t0;
        return;
    }
    // loss |x_target_body - target|^2 and its seed
    const int lb = sc.loss_body;
    const double dx = cur[ADJ_STATE * lb + 0] - sc.target[0], dy = cur[ADJ_STATE * lb + 1] - sc.target[1],
                 dz = cur[ADJ_STATE * lb + 2] - sc.target[2];
    sc.loss[0] = dx * dx + dy * dy + dz * dz;
    double* g = sc.grad_state;  // adjoint of the current state
    for (size_t k = 0; k < stride; ++k) g[k] = 0.0;
    for (int i = 0; i < nb; ++i) { sc.grad_invm[i] = 0.0; sc.grad_mu[2 * i] = 0.0; sc.grad_mu[2 * i + 1] = 0.0; }
    g[ADJ_STATE * lb + 0] = 2.0 * dx;
    g[ADJ_STATE * lb + 1] = 2.0 * dy;
    g[ADJ_STATE * lb + 2] = 2.0 * dz;
    for (int k = 0; k < 6; ++k) sc.prof[k] = 0;
    sc.prof[0] = clock64() - t0;
}

// exclusive scan of a[0, n) in place by a block of TAPE_BLOCK threads
__device__ void block_scan(int* a, int n) {
    __shared__ int s_sum[TAPE_BLOCK / 32], s_run;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_run = 0;
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += TAPE_BLOCK) {
        const int i = i0 + tid, v = i < n ? a[i] : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_sum[warp] = x;
        __syncthreads();
        int base = s_run, all = s_run;
        for (int w = 0; w < TAPE_BLOCK / 32; ++w) {
            if (w < warp) base += s_sum[w];
            all += s_sum[w];
        }
        if (i < n) a[i] = base + x - v;
        __syncthreads();
        if (tid == 0) s_run = all;
    }
    __syncthreads();
}

// One taped substep (block b of scene b / G tapes substep last - b % G of the segment), then its tape put
// in the reverse sweep's order: entries by descending level, and for each the edges to its children in the
// order the tape holds them, so that an adjoint is one sum of a fixed order. The taping is one thread's
// serial work (20 ms for a row of 12 dominoes): the 480 substeps of 24 such rows, one after the other in each
// scene before, took 250 ms and now 38 (three blocks an SM at 168 registers: two waves).
__global__ void __launch_bounds__(TAPE_BLOCK) k_adjoint_tape(const AdjointScene* scenes, const AdjointWorker* workers, AdjointParams P,
                                                             int G, int last) {
    const AdjointScene& sc = scenes[blockIdx.x / G];
    const AdjointWorker& w = workers[blockIdx.x];
    const int u = last - (int)(blockIdx.x % G), tid = threadIdx.x, lane = tid & 31;
    if (u < 0) return;
    const long long t0 = clock64();
    const int nb = sc.nb;
    if (tid == 0) {
        Tape& t = s_tape;
        t.edge = w.edge;
        t.partial = w.partial;
        t.level = w.level;
        t.n = t.m = t.levels = t.overflow = 0;
        t.ncap = w.ncap;
        t.mcap = w.mcap;
        GBody<AVar>* B = reinterpret_cast<GBody<AVar>*>(w.bodies);
        AVar* lam = reinterpret_cast<AVar*>(w.lam);
        GScene<AVar> X;
        X.tv = reinterpret_cast<V3<AVar>*>(w.tv);
        X.tn = reinterpret_cast<V3<AVar>*>(w.tn);
        X.tvv = reinterpret_cast<V3<double>*>(w.tv_val);
        X.tnv = reinterpret_cast<V3<double>*>(w.tn_val);
        X.con = reinterpret_cast<GCon<AVar>*>(w.con);
        X.ncon = 0;
        X.con_cap = sc.contact_cap;
        X.clip = reinterpret_cast<GClip<AVar>*>(w.clip);
        X.epa = reinterpret_cast<GEpa*>(w.epa);
        const int fl = u / P.substeps;
        const double* start = sc.segment + (size_t)u * ADJ_STATE * nb;
        const int2* pairs = sc.pairs + (size_t)fl * sc.pair_cap;
        const uint8_t* active = sc.active_seg + (size_t)fl * nb;
        const double h = P.dt / P.substeps;
        for (int i = 0; i < nb; ++i) {
            g_body(B[i], start, sc, i, active);
            w.stamp[i] = 0;
        }
        for (int i = 0; i < nb; ++i) g_fall(B[i], sc, i, P, h);
        if (P.collisions) {
            const int np = sc.npairs[fl];
            for (int k = 0; k < np; ++k) {
                const int2 p = pairs[k];
                if (g_skip(sc, active, p)) continue;
                if (!w.stamp[p.x]) { g_transform(sc, P.geom, B[p.x], p.x, X, 0, 1); w.stamp[p.x] = 1; }
                if (!w.stamp[p.y]) { g_transform(sc, P.geom, B[p.y], p.y, X, 0, 1); w.stamp[p.y] = 1; }
                g_pair_contacts(sc, P.geom, X, B, p.x, p.y);
            }
        }
        for (int e = 0; e < 4 * sc.ne; ++e) lam[e] = AVar(0.0);
        for (int it = 0; it < P.pos_iters; ++it)
            for (int k = 0; k < sc.ne + X.ncon; ++k) g_node(sc, B, X.con, lam, k, h);
        for (int i = 0; i < nb; ++i) g_velocity(B[i], h);
        for (int c = 0; c < X.ncon; ++c) g_contact_velocity(B[X.con[c].a], B[X.con[c].b], X.con[c], h);
        for (int i = 0; i < nb; ++i) {
            const AVar out[ADJ_STATE] = {B[i].x.x, B[i].x.y, B[i].x.z, B[i].q.x, B[i].q.y, B[i].q.z, B[i].q.w,
                                         B[i].v.x, B[i].v.y, B[i].v.z, B[i].w.x, B[i].w.y, B[i].w.z};
            for (int k = 0; k < ADJ_STATE; ++k) w.out[ADJ_STATE * i + k] = out[k].id;
        }
        if (t.overflow) atomicOr(sc.status, ADJ_ST_TAPE);
    }
    __syncthreads();
    const int n = s_tape.n, m = s_tape.m, L = s_tape.levels;
    for (int l = tid; l <= L; l += TAPE_BLOCK) w.level_start[l] = 0;
    for (int i = tid; i <= n; i += TAPE_BLOCK) w.child_start[i] = 0;
    for (int i = tid; i < n; i += TAPE_BLOCK) w.adj[i] = 0.0;
    __syncthreads();
    for (int i = tid; i < n; i += TAPE_BLOCK) atomicAdd(&w.level_start[L - 1 - w.level[i]], 1);
    __syncthreads();
    block_scan(w.level_start, L + 1);
    for (int l = tid; l < L; l += TAPE_BLOCK) w.cursor[l] = w.level_start[l];
    __syncthreads();
    // an entry's place within its level is free: it changes no sum
    for (int i = tid; i < n; i += TAPE_BLOCK) w.pos[i] = atomicAdd(&w.cursor[L - 1 - w.level[i]], 1);
    __syncthreads();
    bool bad = false;
    for (int e = tid; e < m; e += TAPE_BLOCK) {
        const int2 pc = w.edge[e];
        if (pc.x < 0 || pc.x >= pc.y || pc.y >= n) bad = true;
        else atomicAdd(&w.child_start[w.pos[pc.x]], 1);
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) {
            atomicOr(sc.status, ADJ_ST_BAD_TAPE);
            w.counts[0] = -1;
        }
        return;
    }
    block_scan(w.child_start, n + 1);
    for (int i = tid; i < n; i += TAPE_BLOCK) w.cursor[i] = w.child_start[i];
    __syncthreads();
    if (tid < 32) {
        for (int e0 = 0; e0 < m; e0 += 32) {
            const int e = e0 + lane;
            const bool in = e < m;
            const int2 pc = in ? w.edge[e] : make_int2(0, 0);
            const int p = in ? w.pos[pc.x] : -1, c = in ? w.pos[pc.y] : 0;
            const double d = in ? w.partial[e] : 0.0;
            const unsigned same = __match_any_sync(0xffffffffu, p);
            const int rank = __popc(same & ((1u << lane) - 1u));
            const int base = in ? w.cursor[p] : 0;
            __syncwarp();
            if (in) {
                w.child[base + rank] = c;
                w.child_partial[base + rank] = d;
                if (rank == 0) w.cursor[p] = base + __popc(same);
            }
            __syncwarp();
        }
        if (tid == 0) {
            w.counts[0] = n;
            w.counts[1] = L;
            w.cycles[0] = clock64() - t0;
        }
    }
}

// The reverse sweeps of a group's substeps, last to first, a block per scene: an entry's adjoint is its seed
// plus the sum over its children of their adjoint times the edge's partial, level by level. Entries and edges
// lie in that order, so the block stages them in chunks of whole levels in shared memory, with the adjoints of
// the last ADJ_RING entries (children are mostly near). Four lanes share an entry's children; in a level that
// does not fit a chunk, and in the last one, whose inputs have long lists, a warp does. Bound by the levels'
// latency (some thousands a substep): one thread walking a scalar tape backwards took 410 ms where this takes
// 13 ms (24 rows of 12 dominoes, 20 substeps).
__global__ void __launch_bounds__(REV_BLOCK) k_adjoint_reverse(const AdjointScene* scenes, const AdjointWorker* workers, int G, int last) {
    extern __shared__ double s_dyn[];
    double* ring = s_dyn;                                   // [ADJ_RING]
    double* s_part = ring + ADJ_RING;                       // [CHUNK_EDGES]
    int* s_child = reinterpret_cast<int*>(s_part + CHUNK_EDGES);
    int* s_start = s_child + CHUNK_EDGES;                   // [CHUNK_ENTRIES + 1]
    __shared__ int s_level[REV_BLOCK + 1];
    const AdjointScene& sc = scenes[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, nb = sc.nb;
    long long t0 = clock64(), tape_cycles = 0;
    double* g = sc.grad_state;
    for (int j = 0; j < G && last - j >= 0; ++j) {
        const AdjointWorker& w = workers[blockIdx.x * G + j];
        const int n = w.counts[0], L = w.counts[1];
        if (n < 0) break;   // a corrupt tape (reported)
        double* adj = w.adj;
        for (int k = tid; k < ADJ_STATE * nb; k += REV_BLOCK) {
            const int id = w.out[k];   // (a constant output has no path to the inputs)
            if (id >= 0) atomicAdd(&adj[w.pos[id]], g[k]);
        }
        __syncthreads();
        int l0 = 0;
        while (l0 < L) {
            const int c0 = w.level_start[l0], e0 = w.child_start[c0];
            // the levels that fit a chunk: the ends are monotonic, so the count of fitting ones is their number
            const int l = l0 + tid;
            const int end = l < L ? w.level_start[l + 1] : 0;
            const bool fits = l < L - 1 && end - c0 <= CHUNK_ENTRIES && w.child_start[end] - e0 <= CHUNK_EDGES;
            s_level[tid] = end - c0;
            const int nl = __syncthreads_count(fits);
            if (nl == 0) {
                const int c1 = w.level_start[l0 + 1];
                for (int p = c0 + (tid >> 5); p < c1; p += REV_BLOCK / 32) {
                    double a = 0.0;
                    for (int k = w.child_start[p] + lane; k < w.child_start[p + 1]; k += 32) {
                        const double ac = adj[w.child[k]];
                        if (ac != 0.0) a += ac * w.child_partial[k];
                    }
                    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                    if (lane == 0) {
                        a += adj[p];
                        adj[p] = a;
                        if (p >= c1 - ADJ_RING) ring[p & (ADJ_RING - 1)] = a;
                    }
                }
                __syncthreads();
                ++l0;
                continue;
            }
            const int cn = s_level[nl - 1], c1 = c0 + cn, en = w.child_start[c1] - e0;
            for (int i = tid; i <= cn; i += REV_BLOCK) s_start[i] = w.child_start[c0 + i] - e0;
            for (int i = tid; i < cn; i += REV_BLOCK) ring[(c0 + i) & (ADJ_RING - 1)] = adj[c0 + i];   // seeds
            for (int i = tid; i < en; i += REV_BLOCK) {
                s_child[i] = w.child[e0 + i];
                s_part[i] = w.child_partial[e0 + i];
            }
            const int kept = c1 - ADJ_RING;   // entries below this one have left the ring
            __syncthreads();
            for (int q = 0; q < nl; ++q) {
                const int p0 = q ? s_level[q - 1] : 0, p1 = s_level[q];
                for (int b = p0; b < p1; b += REV_BLOCK / 4) {
                    const int p = b + (tid >> 2);
                    double a = 0.0;
                    if (p < p1)
                        for (int k = s_start[p] + (tid & 3); k < s_start[p + 1]; k += 4) {
                            const int c = s_child[k];
                            const double ac = c >= kept ? ring[c & (ADJ_RING - 1)] : adj[c];
                            if (ac != 0.0) a += ac * s_part[k];
                        }
                    a += __shfl_xor_sync(0xffffffffu, a, 1);
                    a += __shfl_xor_sync(0xffffffffu, a, 2);
                    if (p < p1 && (tid & 3) == 0) ring[(c0 + p) & (ADJ_RING - 1)] += a;
                }
                __syncthreads();
            }
            for (int i = tid; i < cn; i += REV_BLOCK) adj[c0 + i] = ring[(c0 + i) & (ADJ_RING - 1)];
            __syncthreads();
            l0 += nl;
        }
        // inputs: 16 per body, in creation order
        for (int k = tid; k < ADJ_LEAVES * nb; k += REV_BLOCK) {
            const double a = adj[w.pos[k]];
            const int i = k / ADJ_LEAVES, c = k % ADJ_LEAVES;
            if (c < ADJ_STATE) g[ADJ_STATE * i + c] = a;
            else if (c == 13) sc.grad_invm[i] += a;
            else sc.grad_mu[2 * i + c - 14] += a;
        }
        if (tid == 0) {
            sc.prof[4] = max(sc.prof[4], (long long)n);
            sc.prof[5] += n;
            tape_cycles = max(tape_cycles, w.cycles[0]);
        }
        __syncthreads();
    }
    if (tid == 0) {
        sc.prof[2] += tape_cycles;
        sc.prof[3] += clock64() - t0;
    }
}

cudaError_t adjoint_launch(const AdjointScene* scenes, const int* turns, int nturns, const AdjointWorker* workers, int G,
                           const AdjointParams& P, cudaStream_t st, int* launches) {
    const int nscenes = turns[nturns];
    const size_t smem = (size_t)ADJ_RING * 8 + (size_t)CHUNK_EDGES * 12 + (size_t)(CHUNK_ENTRIES + 1) * 4;
    cudaError_t e = cudaFuncSetAttribute(k_adjoint_reverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int K = P.checkpoint_every, nseg = (P.frames + K - 1) / K;
    k_adjoint_forward<<<nscenes, 32 * ADJ_WARPS, 0, st>>>(scenes, P, -1);
    ++*launches;
    for (int seg = nseg - 1; seg >= 0; --seg) {
        if (seg < nseg - 1) {
            k_adjoint_forward<<<nscenes, 32 * ADJ_WARPS, 0, st>>>(scenes, P, seg);
            ++*launches;
        }
        const int nsub = (min(P.frames, (seg + 1) * K) - seg * K) * P.substeps;
        for (int last = nsub - 1; last >= 0; last -= G)
            for (int t = 0; t < nturns; ++t) {
                const int s0 = turns[t], n = turns[t + 1] - s0;
                k_adjoint_tape<<<n * G, TAPE_BLOCK, 0, st>>>(scenes + s0, workers + s0 * G, P, G, last);
                k_adjoint_reverse<<<n, REV_BLOCK, smem, st>>>(scenes + s0, workers + s0 * G, G, last);
                *launches += 2;
            }
    }
    return cudaGetLastError();
}

size_t adjoint_stage_bytes() { return (size_t)ADJ_WARPS * CMAX * sizeof(GCon<double>); }
size_t adjoint_body_bytes(bool tape) { return tape ? sizeof(GBody<AVar>) : sizeof(GBody<double>); }
size_t adjoint_var_bytes() { return sizeof(AVar); }
size_t adjoint_contact_bytes(bool tape) { return tape ? sizeof(GCon<AVar>) : sizeof(GCon<double>); }
size_t adjoint_clip_bytes(bool tape) { return tape ? sizeof(GClip<AVar>) : ADJ_WARPS * sizeof(GClip<double>); }
size_t adjoint_epa_bytes(bool tape) { return (tape ? 1 : ADJ_WARPS) * sizeof(GEpa); }

}  // namespace rp
