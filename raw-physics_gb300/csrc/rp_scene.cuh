// The solver half of a substep for one scene by one CTA, with the scene's state in shared memory.
//
// After the narrowphase a substep is a chain of short phases, each of which depends on all of the one
// before: the schedules of the two Gauss-Seidel sweeps, the position sweep level by level, the velocity
// update, the velocity sweep level by level, the next substep's predict. As kernels of their own, with the
// state in global memory, every solver node waits for six dependent round trips to L2 (about 3500 cycles
// before its first multiply; a contact itself takes about 1000) and the phases for four launches. Here a
// CTA loads its scene's bodies, joints and active nodes once, works in shared memory with block barriers
// between levels, and stores the result once.
//
// Shared memory per body 125 B (FP32 build: pose deltas, orientation, mass properties, friction history;
// the velocities take over the deltas' room after the position sweep), per active node 24 B, per joint
// 104 B. The exact build keeps its bodies in global memory (it is bound by FP64 arithmetic) and stages the
// schedules only. A scene with more active nodes, or more levels, than its room holds is swept
// from global memory by the general code (solve_scene_general).
//
// Measured (GB300; sweeps, velocity update and predict of one substep, before as four kernels -> after): one
// scene of 150 bodies 133 -> 60 us; 96 scenes of up to 512 bodies, a quarter with chains, 754 -> 340 us;
// 768 chains of 33 links 250 -> 94 us.
#pragma once
#include "rp_step.cuh"
#include "rp_launch.h"

namespace rp {

constexpr int SOLVE_BLOCK = 256;        // largest CTA of k_solve
constexpr int SOLVE_LEVELS = 256;       // levels counted in shared memory


// Sizes a launch provides for: bodies, active nodes and joints of its largest scene.
struct SolveRoom {
    int bodies, nodes, joints;
};
__host__ __device__ inline SolveRoom solve_room(int bodies, int joints) {
    // active pairs of a body: resting hulls touch three to six others, each pair counted once
    return SolveRoom{bodies, 2 * bodies + joints + 32, joints};
}
template <typename R>
__host__ __device__ constexpr size_t solve_body_bytes() { return sizeof(R) == 4 ? 7 * 16 : 0; }
template <typename R>
__host__ __device__ inline size_t solve_smem(const SolveRoom& m) {
    size_t b = (size_t)m.nodes * 16 + solve_body_bytes<R>() * (size_t)m.bodies;   // records, body state
    if (sizeof(R) == 4) b += (size_t)m.joints * sizeof(JointF);
    b += (size_t)m.bodies * (8 + 4) + (size_t)m.nodes * 8;                        // level tables and lists
    b += (size_t)m.bodies;                                                        // fixed flags
    return (b + 15) & ~(size_t)15;
}

// An active node of the substep: a joint (pair < 0; body slots of its scene in a, b) or a pair with contacts.
struct __align__(16) NodeRec {
    int pair;              // global pair slot; -1: a joint
    unsigned short a, b;   // scene-local bodies
    int cstart;            // first contact in the contact buffer; joints: index within the scene
    int nc;
};

struct SolveShared {
    int scan[32];
    int cnt[2][SOLVE_LEVELS];   // nodes per level, then the level ends
    int L[2], n, general;
};

// Levels (longest path over shared dynamic bodies, in list order) of the nodes rec[lo, n) by one warp, 32
// nodes at a time: within a chunk each lane finds the last lane before it that touches one of its bodies
// through a per-body mask of the chunk's lanes, the levels of earlier chunks come from a per-body
// table, and the chunk relaxes until nothing changes (once or twice in a heap, a node at a time along a chain).
__device__ __forceinline__ void solve_levels(const NodeRec* rec, const uint8_t* fixed, int lo, int n, unsigned* owner,
                                             unsigned short* blev, unsigned short* lev, SolveShared& sh, int which) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u, above = ~((2u << lane) - 1u);
    int top = 0;
    for (int base = lo; base < n; base += 32) {
        const int i = base + lane;
        int a = -1, b = -1;
        if (i < n) {
            const NodeRec r = rec[i];
            if (!fixed[r.a]) a = r.a;
            if (!fixed[r.b] && r.b != r.a) b = r.b;
        }
        if (a >= 0) atomicOr(&owner[a], 1u << lane);
        if (b >= 0) atomicOr(&owner[b], 1u << lane);
        __syncwarp();
        const unsigned ma = a >= 0 ? owner[a] : 0u, mb = b >= 0 ? owner[b] : 0u;
        int l = 0;
        if (a >= 0) l = blev[a];
        if (b >= 0) l = max(l, (int)blev[b]);
        const int pa = (ma & below) ? 31 - __clz(ma & below) : -1, pb = (mb & below) ? 31 - __clz(mb & below) : -1;
        for (;;) {
            const int la = __shfl_sync(0xffffffffu, l, pa & 31), lb = __shfl_sync(0xffffffffu, l, pb & 31);
            const int m = max(l, max(pa >= 0 ? la + 1 : 0, pb >= 0 ? lb + 1 : 0));
            const bool changed = m != l;
            l = m;
            if (!__any_sync(0xffffffffu, changed)) break;
        }
        const bool live = a >= 0 || b >= 0;
        if (i < n) lev[i] = live ? (unsigned short)min(l, 0xfffe) : 0xffff;
        if (a >= 0 && !(ma & above)) { blev[a] = (unsigned short)min(l + 1, 0xfffe); owner[a] = 0u; }
        if (b >= 0 && !(mb & above)) { blev[b] = (unsigned short)min(l + 1, 0xfffe); owner[b] = 0u; }
        if (live) {
            top = max(top, l + 1);
            if (l < SOLVE_LEVELS) atomicAdd(&sh.cnt[which][l], 1);
            else sh.general = 1;
        }
        __syncwarp();
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) sh.L[which] = min(top, SOLVE_LEVELS);
}

// A sweep of scene s from global memory by the general code, for scenes that outgrow their room: the
// schedules and the position sweeps, or the velocity sweep.
template <typename R, bool EXACT, bool VELOCITY>
__device__ __noinline__ void solve_scene_general(const WorldView<R>& W, int s, double h, int iters) {
    CtaGroup g;
    if (VELOCITY) {
        sweep_levels<R, EXACT, true>(W, g, s, (R)h);
        return;
    }
    const int b0 = W.scene_body[s], b1 = W.scene_body[s + 1];
    if (threadIdx.x == 0) { W.act_count[2 * s] = 0; W.act_count[2 * s + 1] = 0; }
    if constexpr (!EXACT)
        for (int b = b0 + (int)threadIdx.x; b < b1; b += blockDim.x) {
            W.sdx[b] = make_float4(0.f, 0.f, 0.f, 0.f);
            W.sdq[b] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    const int e0 = W.scene_ext[s], e1 = W.scene_ext[s + 1];
    for (int e = 4 * e0 + (int)threadIdx.x; e < 4 * e1; e += blockDim.x) W.ext_lambda[e] = 0.0;
    __syncthreads();
    resched(W, g, s);
    for (int it = 0; it < iters; ++it) sweep_levels<R, EXACT, false>(W, g, s, (R)h);
}

// alike: levels of at most ALIKE_NODES nodes round both bodies of a contact alike (the single large scene's small
// levels, see sweep_levels). predict: the next substep's predict follows (false in a frame's last substep,
// which records the schedules for rp_last_schedule instead); reset: this launch also zeroes the
// next substep's narrowphase counters.
template <typename R, bool EXACT>
__global__ void __launch_bounds__(SOLVE_BLOCK, 2) k_solve(WorldView<R> W, const int32_t* scenes, SolveRoom room, double h, double inv_h, int iters,
                                                          int alike, int predict, int reset) {
    if (frame_abandoned(W.status)) return;
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ SolveShared sh;
    constexpr bool STAGED = !EXACT;
    const int s = scenes[blockIdx.x];
    const int tid = (int)threadIdx.x, nt = (int)blockDim.x;
    const int b0 = W.scene_body[s], nb = W.scene_body[s + 1] - b0;
    const int e0 = W.scene_ext[s], ne = W.scene_ext[s + 1] - e0;
    const int nbase = W.scene_node_cap[s], nn = W.scene_nodes[s], pbase = W.scene_pair_cap[s];
    // shared memory: records, body state, joints, level tables
    NodeRec* rec = reinterpret_cast<NodeRec*>(dyn_smem);
    float4* F = reinterpret_cast<float4*>(rec + room.nodes);
    const int MB = room.bodies;
    float4* s_q = F;                 // orientation: predicted (position sweep), folded (velocity sweep)
    float4* s_dq = F + MB;           // orientation correction; then velocity
    float4* s_dx = F + 2 * MB;       // position correction, inverse mass; then previous angular velocity, inverse mass
    float4* s_S0 = F + 3 * MB;       // inverse inertia xx yy zz xy
    float4* s_S1 = F + 4 * MB;       // inverse inertia xz yz, static and dynamic friction
    float4* s_pd = F + 5 * MB;       // predict displacement, restitution; then angular velocity, restitution
    float4* s_pq = F + 6 * MB;       // previous orientation; then previous velocity
    JointF* joints = reinterpret_cast<JointF*>(F + (STAGED ? 7 * MB : 0));
    unsigned* owner = reinterpret_cast<unsigned*>(joints + (STAGED ? room.joints : 0));   // [2 * bodies]
    unsigned short* blev = reinterpret_cast<unsigned short*>(owner + 2 * MB);             // [2 * bodies]
    unsigned short* lev = blev + 2 * MB;                                                  // [2 * nodes]
    unsigned short* ord = lev + 2 * room.nodes;                                           // [2 * nodes]
    uint8_t* fixed = reinterpret_cast<uint8_t*>(ord + 2 * room.nodes);                    // [bodies]

    if (tid == 0) { sh.n = ne; sh.general = ne > room.joints ? 1 : 0; sh.L[0] = sh.L[1] = 0; }
    for (int l = tid; l < 2 * SOLVE_LEVELS; l += nt) sh.cnt[l / SOLVE_LEVELS][l % SOLVE_LEVELS] = 0;
    for (int b = tid; b < nb; b += nt) {
        const int g = b0 + b;
        fixed[b] = W.fixed[g];
        owner[b] = 0u; owner[MB + b] = 0u;
        blev[b] = 0; blev[MB + b] = 0;
        if constexpr (STAGED) {
            const float4 m = reinterpret_cast<const float4*>(W.material)[g];
            const R* S = W.inv_inertia + 6 * (size_t)g;
            const float4 pd = W.pred_d[g];
            s_q[b] = W.pose_f[2 * g + 1];
            s_dq[b] = make_float4(0.f, 0.f, 0.f, 0.f);
            s_dx[b] = make_float4(0.f, 0.f, 0.f, W.inv_mass[g]);
            s_S0[b] = make_float4(S[0], S[1], S[2], S[3]);
            s_S1[b] = make_float4(S[4], S[5], m.x, m.y);
            s_pd[b] = make_float4(pd.x, pd.y, pd.z, m.z);
            s_pq[b] = W.prev_qf[g];
        }
    }
    // active nodes in constraint order: the joints, then the pairs the contact write-out marked (its bits are
    // cleared for the next substep; a scene's nodes start on a word of their own)
    for (int e = tid; e < ne && ne <= room.joints; e += nt) {
        const ExtConstraint& C = W.ext[e0 + e];
        rec[e] = NodeRec{-1, (unsigned short)(C.e1 - b0), (unsigned short)(C.e2 - b0), e, 0};
        if constexpr (STAGED) joints[e] = load_joint(W, C);
    }
    __syncthreads();
    const int words = (nn + 31) >> 5;
    uint32_t* bits = W.node_bits + (nbase >> 5);
    for (int base = 0; base < words; base += nt) {
        const int w = base + tid;
        uint32_t m = 0;
        if (w < words) { m = bits[w]; bits[w] = 0u; }
        int total;
        int at = block_incl_scan(__popc(m), sh.scan, total) - __popc(m) + sh.n;
        while (m) {
            const int k = (w << 5) + __ffs(m) - 1;
            m &= m - 1u;
            if (at < room.nodes) rec[at].pair = pbase + (k - ne);
            ++at;
        }
        __syncthreads();
        if (tid == 0) sh.n += total;
        __syncthreads();
    }
    const int n = sh.n;
    if (n > room.nodes && tid == 0) sh.general = 1;
    for (int i = ne + tid; i < min(n, room.nodes); i += nt) {
        const int p = rec[i].pair;
        const int2 pr = W.pairs[p];
        rec[i] = NodeRec{p, (unsigned short)(pr.x - b0), (unsigned short)(pr.y - b0), W.scene_contact_cap[s] + W.pair_cstart[p],
                         W.pair_ccount[p]};
    }
    __syncthreads();
    if (!sh.general) {
        const int wid = tid >> 5;
        if (wid == 0) solve_levels(rec, fixed, 0, n, owner, blev, lev, sh, 0);
        if (wid == 1) solve_levels(rec, fixed, ne, n, owner + MB, blev + MB, lev + room.nodes, sh, 1);
        __syncthreads();
    }
    const bool general = sh.general != 0;
    Duo D = duo_of_lane();
    const Oct O = oct_of_lane();
    constexpr int LANES = EXACT ? 8 : 2;   // of a node
    const int nw = nt >> 5, first = (tid & 31) / LANES * nw + (tid >> 5), step = nt / LANES;
    const float4* contacts4 = reinterpret_cast<const float4*>(W.contacts);
    if (general) {
        solve_scene_general<R, EXACT, false>(W, s, h, iters);
        __syncthreads();
    } else {
        // bucket by level: level ends from the counts, then every node takes a place of its level
        if (tid < 64) {
            int* cnt = sh.cnt[tid >> 5];
            const int L = sh.L[tid >> 5];
            int carry = 0;
            for (int base = 0; base < L; base += 32) {
                const int l = base + (tid & 31);
                const int c = l < L ? cnt[l] : 0, incl = warp_incl_scan(c);
                if (l < L) cnt[l] = carry + incl - c;
                carry += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        __syncthreads();
        for (int i = tid; i < n; i += nt) {
            if (lev[i] != 0xffff) ord[atomicAdd(&sh.cnt[0][lev[i]], 1)] = (unsigned short)i;
            if (i >= ne && lev[room.nodes + i] != 0xffff)
                ord[room.nodes + atomicAdd(&sh.cnt[1][lev[room.nodes + i]], 1)] = (unsigned short)i;
        }
        if (tid == 0) atomicAdd(&W.counters[6], (unsigned long long)sh.L[0]);
        __syncthreads();
        if (!predict) {   // the frame's last substep: the schedules rp_last_schedule reports
            for (int which = 0; which < 2; ++which) {
                const SchedView<R> v = sched_view(W, s, which);
                const int L = sh.L[which];
                // zero beyond L up to the levels of the schedule recorded before: resched counts on it
                const int used = max(L, min(*(volatile int*)v.levels + 1, W.max_levels));
                for (int l = tid; l <= used; l += nt) { v.count[l] = l && l <= L ? sh.cnt[which][l - 1] : 0; v.fill[l] = 0; }
                const int m = L ? sh.cnt[which][L - 1] : 0;
                for (int i = tid; i < m; i += nt) {
                    const int r = ord[which * room.nodes + i];
                    v.nodes[i] = rec[r].pair < 0 ? r : rec[r].pair - pbase + ne;
                }
                __syncthreads();
                if (tid == 0) *v.levels = L;
            }
        }
        // lane pairs (exact build: eight lanes) take a level's nodes, consecutive nodes in different warps (a warp runs as long as its
        // longest node)
        for (int it = 0; it < iters; ++it) {
            int lo = 0;
            for (int l = 0; l < sh.L[0]; ++l) {
                const int hi = sh.cnt[0][l];
                if (alike) D.second_right = D.side != 0 && hi - lo > ALIKE_NODES;
                for (int i = lo + first; i < hi; i += step) {
                    const NodeRec r = rec[ord[i]];
                    if constexpr (EXACT) {
                        if (r.pair < 0) {
                            double* lam = W.ext_lambda + 4 * (size_t)(e0 + r.cstart);
                            if (it == 0 && O.lead()) { lam[0] = 0.0; lam[1] = 0.0; lam[2] = 0.0; }
                            __syncwarp(O.oct);
                            ext_solve(W, O, W.ext[e0 + r.cstart], lam, h);
                        } else {
                            dsolve_pair(W, O, b0 + (O.side ? r.b : r.a), W.contacts + 12 * (size_t)r.cstart, r.nc, h);
                        }
                    } else {
                        const int me = D.side ? r.b : r.a;
                        FBody B;
                        {
                            const float4 q = s_q[me], dq = s_dq[me], dx = s_dx[me], S0 = s_S0[me], S1 = s_S1[me];
                            B.q0f = qt<float>(q.x, q.y, q.z, q.w);
                            B.dq = qt<float>(dq.x, dq.y, dq.z, dq.w);
                            B.dx = v3<float>(dx.x, dx.y, dx.z);
                            B.invm = dx.w;
                            B.S[0] = S0.x; B.S[1] = S0.y; B.S[2] = S0.z; B.S[3] = S0.w; B.S[4] = S1.x; B.S[5] = S1.y;
                            B.fixed = fixed[me] != 0;
                            B.idx = me;
                        }
                        if (r.pair < 0) {
                            float l3[3] = {0.f, 0.f, 0.f};
                            float* lam = reinterpret_cast<float*>(W.ext_lambda + 4 * (size_t)(e0 + r.cstart));
                            if (it > 0) { l3[0] = lam[0]; l3[1] = lam[1]; l3[2] = lam[2]; }
                            __syncwarp(D.mask);
                            fext_solve(D, B, W.rot + b0 + me, joints[r.cstart], l3, (float)h);
                            if (it + 1 < iters && D.side == 0) { lam[0] = l3[0]; lam[1] = l3[1]; lam[2] = l3[2]; }
                        } else {
                            const float mus_own = s_S1[me].z;
                            const float mus = __fadd_rn(mus_own, D.other(mus_own)) / 2.0f;
                            const float4 bb = W.pair_base[r.pair];
                            const float4* c4 = contacts4 + 3 * (size_t)r.cstart;
                            float4 rl = c4[D.side], nn4 = c4[2];
                            const V3<float> base = D.own(v3<float>(bb.x, bb.y, bb.z));
                            for (int c = 0; c < r.nc; ++c) {
                                const float4 r0 = rl;
                                const V3<float> nv = D.own(v3<float>(nn4.x, nn4.y, nn4.z));
                                if (c + 1 < r.nc) { rl = c4[3 * (c + 1) + D.side]; nn4 = c4[3 * (c + 1) + 2]; }
                                const float lam = fcollision_solve(s_pd, s_pq, D, B, base, r0, nv, mus);
                                if (lam != r0.w) W.contacts[12 * ((size_t)r.cstart + c) + 4 * D.side + 3] = (R)lam;
                            }
                        }
                        if (!B.fixed) {
                            s_dx[me] = make_float4(B.dx.x, B.dx.y, B.dx.z, B.invm);
                            s_dq[me] = make_float4(B.dq.x, B.dq.y, B.dq.z, B.dq.w);
                        }
                    }
                }
                lo = hi;
                __syncthreads();
            }
        }
    }
    // velocity update: the corrections into the FP64 pose, then the velocities of awake bodies from it
    if constexpr (EXACT) {
        for (int b = tid >> 2; b < nb; b += nt >> 2) oct_velocity(W, O, b0 + b, inv_h);
    } else for (int b = tid; b < nb; b += nt) {
        const int g = b0 + b;
        double4_32a p = W.pos[g], q = W.rot[g];
        const double4_32a pp = W.prev_pos[g], pq = W.prev_rot[g];
        const bool moves = !fixed[b] && W.active[g];
        V3<R> v = v3<R>(W.vel[3 * g], W.vel[3 * g + 1], W.vel[3 * g + 2]);
        V3<R> w = v3<R>(W.omega[3 * g], W.omega[3 * g + 1], W.omega[3 * g + 2]);
        V3<R> pv = v3<R>(W.prev_vel[3 * g], W.prev_vel[3 * g + 1], W.prev_vel[3 * g + 2]);
        V3<R> pw = v3<R>(W.prev_omega[3 * g], W.prev_omega[3 * g + 1], W.prev_omega[3 * g + 2]);
        const float4 dx = general ? W.sdx[g] : s_dx[b], dq = general ? W.sdq[g] : s_dq[b];
        if (fold_pose(p, q, dx, dq)) {
            W.pos[g] = p;
            W.rot[g] = q;
            s_q[b] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
        }
        if (general) W.pose_f[2 * g + 1] = s_q[b];
        if (moves) {
            pv = v;
            pw = w;
            W.prev_vel[3 * g] = v.x; W.prev_vel[3 * g + 1] = v.y; W.prev_vel[3 * g + 2] = v.z;
            W.prev_omega[3 * g] = w.x; W.prev_omega[3 * g + 1] = w.y; W.prev_omega[3 * g + 2] = w.z;
            velocity_values<R, EXACT>(p, q, pp, pq, inv_h, v, w);
            if (general) {   // otherwise stored after the velocity sweep
                W.vel[3 * g] = v.x; W.vel[3 * g + 1] = v.y; W.vel[3 * g + 2] = v.z;
                W.omega[3 * g] = w.x; W.omega[3 * g + 1] = w.y; W.omega[3 * g + 2] = w.z;
            }
        }
        s_dq[b] = make_float4(v.x, v.y, v.z, 0.f);
        s_pd[b] = make_float4(w.x, w.y, w.z, s_pd[b].w);
        s_pq[b] = make_float4(pv.x, pv.y, pv.z, 0.f);
        s_dx[b] = make_float4(pw.x, pw.y, pw.z, s_dx[b].w);
    }
    __syncthreads();
    if (general) {
        solve_scene_general<R, EXACT, true>(W, s, h, iters);
        __syncthreads();
    } else {
        int lo = 0;
        for (int l = 0; l < sh.L[1]; ++l) {
            const int hi = sh.cnt[1][l];
            for (int i = lo + first; i < hi; i += step) {
                const NodeRec r = rec[ord[room.nodes + i]];
                const int me = (EXACT ? O.side : D.side) ? r.b : r.a;
                if constexpr (EXACT) {
                    dvsolve_pair(W, O, b0 + me, W.contacts + 12 * (size_t)r.cstart, r.nc, h);
                } else {
                    const float4* c4 = contacts4 + 3 * (size_t)r.cstart;
                    float4 rl = c4[D.side], nn4 = c4[2];
                    const float4 q4 = s_q[me], v4 = s_dq[me], w4 = s_pd[me], pv4 = s_pq[me], pw4 = s_dx[me], S0 = s_S0[me], S1 = s_S1[me];
                    const float S[6] = {S0.x, S0.y, S0.z, S0.w, S1.x, S1.y};
                    const Qt<float> q = qt<float>(q4.x, q4.y, q4.z, q4.w);
                    const M3<float> I = world_tensor_f(q, S);
                    const bool fx = fixed[me] != 0;
                    V3<float> v = v3<float>(v4.x, v4.y, v4.z), w = v3<float>(w4.x, w4.y, w4.z);
                    const V3<float> pv = v3<float>(pv4.x, pv4.y, pv4.z), pw = v3<float>(pw4.x, pw4.y, pw4.z);
                    const float mud = __fadd_rn(S1.w, D.other(S1.w)) / 2.0f;
                    const float e = __fmul_rn(w4.w, D.other(w4.w));
                    for (int c = 0; c < r.nc; ++c) {
                        const float4 r0 = rl, n0 = nn4;
                        if (c + 1 < r.nc) { rl = c4[3 * (c + 1) + D.side]; nn4 = c4[3 * (c + 1) + 2]; }
                        const float lother = D.other(r0.w);
                        const V3<float> rr = rotate_f(q, v3<float>(r0.x, r0.y, r0.z), true);
                        fcontact_velocity(D, rr, I, D.own(v3<float>(n0.x, n0.y, n0.z)), pw4.w, fx, D.first(r0.w, lother), (float)h, mud, e, v, w,
                                          pv, pw);
                    }
                    if (!fx) {
                        s_dq[me] = make_float4(v.x, v.y, v.z, 0.f);
                        s_pd[me] = make_float4(w.x, w.y, w.z, w4.w);
                    }
                }
            }
            lo = hi;
            __syncthreads();
        }
        if constexpr (STAGED) {
            for (int b = tid; b < nb; b += nt) {
                const int g = b0 + b;
                if (fixed[b]) continue;
                const float4 v = s_dq[b], w = s_pd[b];
                W.vel[3 * g] = v.x; W.vel[3 * g + 1] = v.y; W.vel[3 * g + 2] = v.z;
                W.omega[3 * g] = w.x; W.omega[3 * g + 1] = w.y; W.omega[3 * g + 2] = w.z;
            }
        }
    }
    // the next substep's counters and predict
    if (!predict) return;
    if (tid == 0) W.contact_count[s] = 0;
    if (reset && blockIdx.x == 0 && tid == 0) reset_narrow_queue(W);
    if constexpr (EXACT) {
        for (int b = tid >> 2; b < nb; b += nt >> 2) oct_predict(W, O, b0 + b, h);
    } else {
        for (int b = tid; b < nb; b += nt) predict_body<R, EXACT, true, false>(W, b0 + b, h);
    }
}

}  // namespace rp
