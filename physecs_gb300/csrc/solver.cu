// solver.cu — contact rows, graph colouring, joint rows and the TGS substep loop.
//
// Restates Physecs src/Physecs.cpp:209-531 with src/ContactConstraints.cpp,
// src/Constraint1D.cpp (scalar rows, joint colour 8) and src/Constraint1DW.cpp
// (4-lane rows, joint colours 0-7).  The reference solves every contact serially;
// here contacts are graph-coloured so that each colour is body-disjoint and its
// contacts can be solved in parallel with a result identical to any serial order
// of that colour.  Joints keep the reference's own colouring (colours 0-7 are
// entity-disjoint); the overflow colour is split into sub-colours on the host.
//
// One persistent kernel runs a whole frame of a scene: colouring, then every
// substep's row update, velocity integration, preSolve, iterations, position
// integration, relaxation and write-back.  Small scenes run one per CTA with
// __syncthreads between phases; large scenes run on a cluster, or on the whole grid,
// where bodies count their finished solves and contacts wait for their turn on both of
// theirs (solve_flow), with grid barriers between phases.  Every wait is bounded.
#include <cooperative_groups.h>
#include "libm_f32.cuh"
#include "smem_limit.cuh"
#include "solver_words.cuh"
#include <algorithm>
#include "frame.cuh"

namespace psx {

constexpr float kPi = 3.14159265358979323846f;

// ---------------------------------------------------------------- restitution cache


// before the contacts: this frame's cache table empty, the counters zero
__global__ void k_contacts_begin(FrameBuf f, int n_scenes) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *f.n_points = 0;
    if (i <= n_scenes) f.man_scene_cnt[i] = 0;
    if (i >= f.cache_cap) return;
    CacheEntry* cur = f.cache_parity[0] ? f.cache_b : f.cache_a;
    cur[i].key = kEmpty;
}

// ---------------------------------------------------------------- contact rows (src/Physecs.cpp:215-314)

// One thread per pair with manifolds.  Fewer than half of the pairs have any, and each is a
// chain of dependent loads, so a warp first lists those of 128 pairs (32 where there are few)
// and then takes them with full lanes; what it adds to the counts goes out once a round and a
// scene.  4096 scenes: 880 us with a thread per pair and an atomic per contact on the world's
// one count of points, 432 now; 256 scenes 90 and 56.
constexpr int kContactThreads = 128, kContactChunk = 128;
__global__ void __launch_bounds__(kContactThreads) k_build_contacts(World w, FrameBuf f) {
    __shared__ int s_list[kContactThreads / 32][kContactChunk];
    int* const list = s_list[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    int np = *f.n_pairs;
    CacheEntry* cur = f.cache_parity[0] ? f.cache_b : f.cache_a;
    const CacheEntry* prev = f.cache_parity[0] ? f.cache_a : f.cache_b;
    unsigned mask = (unsigned)f.cache_cap - 1u;
    const int chunk = np >= warps * kContactChunk ? kContactChunk : 32;
    int points = 0;
    for (int base = warp * chunk; base < np; base += warps * chunk) {
        int listed = 0;
        for (int at = base; at < min(base + chunk, np); at += 32) {
            const unsigned m = __ballot_sync(~0u, at + lane < np && f.pair_nman[at + lane]);
            if (m >> lane & 1) list[listed + __popc(m & ((1u << lane) - 1u))] = at + lane;
            listed += __popc(m);
        }
        __syncwarp();
        for (int i0 = 0; i0 < listed; i0 += 32) {
            int scene = -1, made = 0;
            if (i0 + lane < listed) {
                const int p = list[i0 + lane], cnt = f.pair_nman[p];
                int off = f.pair_moff[p];
                int2 pr = f.pairs[p];
                int4 cA = w.col_info[pr.x], cB = w.col_info[pr.y];
                int bodyA = cA.x, bodyB = cB.x;
                int4 iA = w.info[bodyA], iB = w.info[bodyB];
                bool simA = (iA.y & BODY_DYN) && !(iA.y & BODY_KIN), simB = (iB.y & BODY_DYN) && !(iB.y & BODY_KIN);
                Q4 qA = ld4(w.quat[bodyA]), qB = ld4(w.quat[bodyB]);
                V3 com0 = {0, 0, 0}, v0 = {0, 0, 0}, w0 = {0, 0, 0}, com1 = {0, 0, 0}, v1 = {0, 0, 0}, w1 = {0, 0, 0};
                if (simA) { com0 = ld3(w.pos[bodyA]) + qrot(qA, ld3(w.com[iA.z])); v0 = ld3(w.vel[iA.z]); w0 = ld3(w.ang[iA.z]); }
                if (simB) { com1 = ld3(w.pos[bodyB]) + qrot(qB, ld3(w.com[iB.z])); v1 = ld3(w.vel[iB.z]); w1 = ld3(w.ang[iB.z]); }
                float4 mA = w.col_mat[pr.x], mB = w.col_mat[pr.y];
                float friction = (mA.x + mB.x) * 0.5f;
                bool soft;
                float freq = 0, damp = 0, rest = 0;
                if (mA.z || mB.z) {
                    soft = true;
                    if (mA.z && mB.z) { freq = fminG(mA.y, mB.y); damp = fminG(mA.z, mB.z); }
                    else if (mA.z) { freq = mA.y; damp = mA.z; }
                    else { freq = mB.y; damp = mB.z; }
                } else {
                    soft = false;
                    rest = (mA.y + mB.y) * 0.5f;
                }
                Q4 iqA = qinverse(qA), iqB = qinverse(qB);
                bool tri = f.pair_cat[p] == 2;
                for (int k = 0; k < cnt; ++k) {
                    int idx = off + k;
                    if (idx >= f.man_cap) { atomicOr(w.err, ERR_MANIFOLD_CAPACITY); break; }
                    const Manifold& m = tri ? f.man_tri[f.pair_tslot[p] * kTriManifolds + k] : f.man_pair[p];
                    Contact c;
                    c.b0 = simA ? iA.z : -1;
                    c.b1 = simB ? iB.z : -1;
                    c.body0 = bodyA; c.body1 = bodyB;
                    V3 n = ld3(m.n);
                    c.n = st4(n, friction);
                    c.frequency = freq; c.damping = damp;
                    c.np = m.np; c.soft = soft ? 1 : 0;
                    c.color = -1; c.scene = iA.w; c.pair = p; c.tri = m.tri;
                    unsigned long long key = cache_key(pr.x, pr.y, m.tri, w.key_cbits);
                    // previous frame's entry, if any
                    const CacheEntry* pe = nullptr;
                    const bool fresh = w.scene_fresh && w.scene_fresh[iA.w];
                    for (unsigned h = cache_hash(key) & mask, probe = 0; !fresh && probe < (unsigned)f.cache_cap; ++probe, h = (h + 1) & mask) {
                        unsigned long long kk = prev[h].key;
                        if (kk == key) { pe = &prev[h]; break; }
                        if (kk == kEmpty) break;
                    }
                    CacheEntry ne;
                    ne.key = key; ne.np = m.np;
                    for (int q = 0; q < m.np; ++q) {
                        V3 r0 = ld3(m.p0[q]) - com0;
                        V3 r1 = ld3(m.p1[q]) - com1;
                        V3 rel = v1 + cross(w1, r1) - v0 - cross(w0, r0);
                        float relN = dot(rel, n);
                        r0 = qrot(iqA, r0);
                        r1 = qrot(iqB, r1);
                        float tv = 0;
                        bool found = false;
                        if (pe) {
                            for (int i = 0; i < pe->np; ++i) {
                                float4 e = pe->r0tv[i];
                                if ((double)distance(r0, ld3(e)) < 0.1) { found = true; tv = e.w; break; }
                            }
                        }
                        if (!found) tv = -rest * relN;
                        ne.r0tv[q] = st4(r0, tv);
                        ContactPt& cp = c.p[q];
                        cp.r0 = st4(r0, tv);
                        cp.r1 = st4(r1, 0.f);
                    }
                    // insert into this frame's table
                    bool placed = false;
                    for (unsigned h = cache_hash(key) & mask, probe = 0; probe < (unsigned)f.cache_cap; ++probe, h = (h + 1) & mask) {
                        unsigned long long old = atomicCAS(&cur[h].key, kEmpty, key);
                        if (old == kEmpty || old == key) {
                            cur[h].np = ne.np;
                            for (int q = 0; q < ne.np; ++q) cur[h].r0tv[q] = ne.r0tv[q];
                            placed = true;
                            break;
                        }
                    }
                    if (!placed) atomicOr(w.err, ERR_CACHE_CAPACITY);
                    f.contacts[idx] = c;
                    ++made;
                    points += m.np;
                }
                scene = iA.w;
            }
            __syncwarp();
            const int first = __shfl_sync(~0u, scene, 0);   // lane 0 has a pair
            if (__all_sync(~0u, scene == first || scene < 0)) {
                made = __reduce_add_sync(~0u, made);
                if (lane == 0 && made) atomicAdd(&f.man_scene_cnt[first], made);
            } else if (made) {
                atomicAdd(&f.man_scene_cnt[scene], made);
            }
        }
        __syncwarp();
    }
    points = __reduce_add_sync(~0u, points);
    if (lane == 0 && points) atomicAdd(f.n_points, points);
}

// ---------------------------------------------------------------- joints

// The rows of schedule entry q (types.cuh): row k, field f at [(k * kRowF4 + f) * 32].
__device__ __forceinline__ float4* joint_rows(const World& w, int q) {
    return w.rows + (size_t)(q >> 5) * (kMaxRowsPerJoint * kRowF4 * 32) + (q & 31);
}
constexpr int kRowStep = kRowF4 * 32;

// getSolverDesc of each joint type (src/Joints/*.cpp): row flags in creation order,
// evaluated at frame start; the prismatic limit row exists only while violated.
__global__ void k_joint_layout(World w, int* n_rows) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= w.n_joints) return;
    const int j = w.jsched[q];
    JointDev J = w.joints[j];
    int f[kMaxRowsPerJoint];
    int n = 0;
    auto add = [&](int fl, int cnt) { for (int i = 0; i < cnt; ++i) f[n++] = fl; };
    enum { RN = 0, RS = 1, RA = 2, RL = 4 };
    switch (J.type) {
        case 0: add(RN, 3); add(RA, 3); break;                                        // fixed
        case 1: add(RN, 3); add(RA, 2); if (J.params[0] != 0.f) add(RA | RL, 1); break;  // revolute
        case 2: add(RN, 3); break;                                                    // spherical
        case 3: {                                                                     // prismatic
            V3 p0 = ld3(w.pos[J.body0]) + qrot(ld4(w.quat[J.body0]), ld3(J.a0p));
            V3 p1 = ld3(w.pos[J.body1]) + qrot(ld4(w.quat[J.body1]), ld3(J.a1p));
            V3 d = p1 - p0;
            V3 u00 = qrot(qmul(ld4(w.quat[J.body0]), ld4(J.a0q)), {1, 0, 0});
            float dx = dot(d, u00);
            add(RN, 2); add(RA, 3);
            if (dx > J.params[0]) { J.makeUpper = 1; J.makeLower = 0; add(RL, 1); }
            else if (dx < J.params[1]) { J.makeUpper = 0; J.makeLower = 1; add(RL, 1); }
            else { J.makeUpper = 0; J.makeLower = 0; }
            if (J.params[2] != 0.f) add(RS, 1);
            break;
        }
        case 4: add(RN, 3); add(RA, 1); break;                                        // universal
        case 5: add(RA, 1); break;                                                    // gear
        default: add(RN, 3); add(RA, 2); add(RA | RS, 1); break;                      // servo
    }
    J.nrows = n;
    atomicAdd(n_rows, n);
    for (int i = 0; i < kMaxRowsPerJoint; ++i) J.rowflags[i] = i < n ? f[i] : -1;
    w.joints[j].makeUpper = J.makeUpper;
    w.joints[j].makeLower = J.makeLower;
    w.joints[j].nrows = n;
    for (int i = 0; i < kMaxRowsPerJoint; ++i) w.joints[j].rowflags[i] = J.rowflags[i];
    // preSolve and solve take the rows by kind, in this order of their flags
    unsigned place = 0;
    int taken = 0;
    const int kinds[6] = {RN, RA, RS, RL, RA | RS, RA | RL};
    float4* const R = joint_rows(w, q);
    for (int kind : kinds)
        for (int i = 0; i < n; ++i) {
            if (J.rowflags[i] != kind) continue;
            place |= (unsigned)taken << (4 * i);
            float4* const r = R + taken++ * kRowStep;
            r[32 * ROW_LINEAR] = make_float4(0, 0, 0, 0);
            r[32 * ROW_ANGULAR0] = make_float4(0, 0, 0, 0);
            r[32 * ROW_ANGULAR1] = make_float4(0, 0, 0, -FLT_MAX);
            r[32 * ROW_ANGULAR0T] = make_float4(0, 0, 0, __int_as_float(kind));
            r[32 * ROW_ANGULAR1T] = make_float4(0, 0, 0, 0);
            r[32 * ROW_MISC] = make_float4(FLT_MAX, 0, 0, 0);
        }
    w.joints[j].place = place;
    w.jruns[q] = JointRun{J.b0, J.b1, n | J.simd << 8, J.b0 >= 0 ? w.com[J.b0].w : 0.f, J.b1 >= 0 ? w.com[J.b1].w : 0.f,
                          J.rank0, J.rank1, 0};
}

int launch_joint_layout(const World& w, FrameBuf& f, cudaStream_t s) {
    cudaMemsetAsync(f.n_rows, 0, sizeof(int), s);
    if (!w.n_joints) return 0;
    k_joint_layout<<<(w.n_joints + 127) / 128, 128, 0, s>>>(w, f.n_rows);
    return 1;
}

__device__ __forceinline__ float angleDiffD(float a0, float a1) {  // GearJoint.cpp:5-8
    const float pi = kPi, two_pi = 6.28318530717958647692f;
    float diff = fmodf(a1 - a0 + pi, two_pi) - pi;
    return diff < -pi ? diff + two_pi : diff;
}

// makeConstraints of each joint type (src/Joints/*.cpp, src/JointsUtil.h:8-28) for schedule
// entry q, rows taken in creation order
__device__ void make_joint_rows(const World& w, int q) {
    JointDev& J = w.joints[w.jsched[q]];
    Q4 q0 = ld4(w.quat[J.body0]), q1 = ld4(w.quat[J.body1]);
    M3 u0 = mat3_cast(qmul(q0, ld4(J.a0q))), u1 = mat3_cast(qmul(q1, ld4(J.a1q)));
    V3 r0 = qrot(q0, ld3(J.r0)), r1 = qrot(q1, ld3(J.r1));
    V3 p0 = ld3(w.pos[J.body0]) + qrot(q0, ld3(J.a0p)), p1 = ld3(w.pos[J.body1]) + qrot(q1, ld3(J.a1p));
    float4* const R = joint_rows(w, q);
    const unsigned place = J.place;
    int k = 0;
    auto row = [&]() { return R + ((place >> (4 * k)) & 15u) * kRowStep; };
    auto lin = [&](V3 l, V3 a0, V3 a1, float c, float lo = -FLT_MAX) {
        float4* const r = row();
        r[32 * ROW_LINEAR] = st4(l, 0.f); r[32 * ROW_ANGULAR0] = st4(a0, c); r[32 * ROW_ANGULAR1] = st4(a1, lo); ++k;
    };
    auto ang = [&](V3 a0, V3 a1, float c) {
        float4* const r = row();
        r[32 * ROW_ANGULAR0] = st4(a0, c); r[32 * ROW_ANGULAR1] = st4(a1, -FLT_MAX); ++k;
    };
    auto p2p = [&]() {
        V3 d = p1 - p0;
        lin({1, 0, 0}, {0, r0.z, -r0.y}, {0, r1.z, -r1.y}, d.x);
        lin({0, 1, 0}, {-r0.z, 0, r0.x}, {-r1.z, 0, r1.x}, d.y);
        lin({0, 0, 1}, {r0.y, -r0.x, 0}, {r1.y, -r1.x, 0}, d.z);
    };
    auto angs = [&](V3 a, float c) { ang(a, a, c); };
    switch (J.type) {
        case 0:
            p2p();
            angs(cross(u1.c[1], u0.c[0]), dot(u0.c[0], u1.c[1]));
            angs(cross(u1.c[2], u0.c[0]), dot(u0.c[0], u1.c[2]));
            angs(cross(u1.c[2], u0.c[1]), dot(u0.c[1], u1.c[2]));
            break;
        case 2: p2p(); break;
        case 4:
            p2p();
            angs(cross(u1.c[2], u0.c[2]), dot(u0.c[2], u1.c[2]));
            break;
        case 1:
            p2p();
            angs(cross(u1.c[1], u0.c[0]), dot(u0.c[0], u1.c[1]));
            angs(cross(u1.c[2], u0.c[0]), dot(u0.c[0], u1.c[2]));
            if (J.params[0] != 0.f) {
                float4* const r = row();
                r[32 * ROW_ANGULAR0] = st4(u0.c[0], 0.f);
                r[32 * ROW_ANGULAR1] = st4(u0.c[0], -J.params[2]);
                r[32 * ROW_LINEAR].w = J.params[1];
                r[32 * ROW_MISC].x = J.params[2];
                ++k;
            }
            break;
        case 6: {
            p2p();
            angs(cross(u1.c[1], u0.c[0]), dot(u0.c[0], u1.c[1]));
            angs(cross(u1.c[2], u0.c[0]), dot(u0.c[0], u1.c[2]));
            float a = libm::acosf(clampG(dot(u0.c[2], u1.c[2]), -1.f, 1.f));   // glm::orientedAngle
            if (dot(u0.c[0], cross(u0.c[2], u1.c[2])) < 0.f) a = -a;
            row()[32 * ROW_MISC].y = J.params[1];
            row()[32 * ROW_MISC].z = J.params[2];
            angs(u0.c[0], a - J.params[0]);
            break;
        }
        case 3: {
            V3 d = p1 - p0;
            lin(u0.c[1], cross(r0, u0.c[1]), cross(r1, u0.c[1]), dot(d, u0.c[1]));
            lin(u0.c[2], cross(r0, u0.c[2]), cross(r1, u0.c[2]), dot(d, u0.c[2]));
            angs(cross(u1.c[1], u0.c[0]), dot(u0.c[0], u1.c[1]));
            angs(cross(u1.c[2], u0.c[0]), dot(u0.c[0], u1.c[2]));
            angs(cross(u1.c[2], u0.c[1]), dot(u0.c[1], u1.c[2]));
            float dx = dot(d, u0.c[0]);
            V3 r0xx = cross(r0, u0.c[0]), r1xx = cross(r1, u0.c[0]);
            if (J.makeUpper) {
                lin(u0.c[0], r0xx, r1xx, dx - J.params[0], 0.f);   // min = 0
            } else if (J.makeLower) {
                row()[32 * ROW_MISC].x = 0.f;  // max = 0
                lin(u0.c[0], r0xx, r1xx, dx - J.params[1]);
            }
            if (J.params[2] != 0.f) {
                row()[32 * ROW_MISC].y = J.params[4];
                row()[32 * ROW_MISC].z = J.params[5];
                lin(u0.c[0], r0xx, r1xx, dx - J.params[3]);
            }
            break;
        }
        default: {  // gear (GearJoint.cpp:10-50)
            float a0, a1;
            {
                V3 p1p = p1 + dot(p0 - p1, u0.c[0]) * u0.c[0];
                V3 dir = normalize(p0 - p1p);
                V3 n = cross(u0.c[0], dir);
                M3 t = mm(transpose(m3cols(u0.c[0], -n, dir)), u0);
                a0 = libm::atan2f(at(t.c[1], 2), at(t.c[2], 2));
            }
            {
                V3 p0p = p0 + dot(p1 - p0, u1.c[0]) * u1.c[0];
                V3 dir = normalize(p0p - p1);
                V3 n = cross(u1.c[0], dir);
                M3 t = mm(transpose(u1), m3cols(u1.c[0], -n, dir));
                a1 = libm::atan2f(at(t.c[1], 2), at(t.c[2], 2));
            }
            if (!J.gearInit) { J.persistent0 = a0; J.persistent1 = a1; J.gearInit = 1; }
            J.virtual0 += angleDiffD(a0, J.persistent0);
            J.virtual1 += angleDiffD(a1, J.persistent1);
            J.persistent0 = a0; J.persistent1 = a1;
            float ratio = J.params[0];
            ang(u0.c[0] * ratio, -u1.c[0], J.virtual0 * ratio - J.virtual1);
            break;
        }
    }
}

// Constraint1D(W)::preSolve (Constraint1D.cpp:5-52 / Constraint1DW.cpp:5-115) of a joint's
// rows in solve order.  Every row of a joint has its two bodies, whose inertia is read once
// and whose pseudo velocities (with the count of rows applied) stay in registers.
__device__ __forceinline__ void joint_rows_presolve(const World& w, int q, float4& pv0, float4& pw0, float4& pv1, float4& pw1) {
    const JointRun J = w.jruns[q];
    float4* R = joint_rows(w, q);
    const int b0 = J.b0, b1 = J.b1, n = J.rows & 0xff;
    const bool simd = (J.rows >> 8) != 0, same = b0 >= 0 && b0 == b1;
    const float im0 = J.im0, im1 = J.im1;
    M3 I0 = m3zero(), I1 = m3zero();
    if (b0 >= 0) I0 = m3cols(ld3(w.mt[3 * b0]), ld3(w.mt[3 * b0 + 1]), ld3(w.mt[3 * b0 + 2]));
    if (b1 >= 0) I1 = m3cols(ld3(w.mt[3 * b1]), ld3(w.mt[3 * b1 + 1]), ld3(w.mt[3 * b1 + 2]));
    for (int i = 0; i < n; ++i, R += kRowStep) {
        const float4 rl = R[32 * ROW_LINEAR], r0 = R[32 * ROW_ANGULAR0], r1 = R[32 * ROW_ANGULAR1];
        const float fw = R[32 * ROW_ANGULAR0T].w, mx = R[32 * ROW_MISC].x;
        const int fl = __float_as_int(fw);
        const bool angf = fl & 2, soft = fl & 1, lim = fl & 4;
        const V3 a0 = ld3(r0), a1 = ld3(r1), l = ld3(rl);
        const V3 a0t = mv(I0, a0), a1t = mv(I1, a1);
        float inv = dot(a0, a0t) + dot(a1, a1t);
        if (!angf) inv += dot(l, l) * (im0 + im1);
        const V3 l0t = im0 * l, l1t = im1 * l;
        const float c = r0.w, mn = r1.w;
        R[32 * ROW_ANGULAR0T] = st4(a0t, fw);
        R[32 * ROW_ANGULAR1T] = st4(a1t, inv);
        if (soft || !(inv != 0.f && c != 0.f)) continue;
        float lambda = c / inv;
        if (lim) {
            if (simd) { lambda = lambda > mn ? lambda : mn; lambda = lambda < mx ? lambda : mx; }
            else lambda = clampG(lambda, mn, mx);
        }
        if (b0 >= 0) {
            pv0 = st4(angf ? ld3(pv0) : ld3(pv0) + lambda * l0t, pv0.w + 1.f);
            pw0 = st4(ld3(pw0) + lambda * a0t, 0.f);
        }
        if (same) { pv1 = pv0; pw1 = pw0; }
        if (b1 >= 0) {
            pv1 = st4(angf ? ld3(pv1) : ld3(pv1) - lambda * l1t, pv1.w + 1.f);
            pw1 = st4(ld3(pw1) - lambda * a1t, 0.f);
        }
        if (same) { pv0 = pv1; pw0 = pw1; }
    }
}

__device__ void joint_presolve(const World& w, int q) {
    const int b0 = w.jruns[q].b0, b1 = w.jruns[q].b1;
    float4 pv0 = make_float4(0, 0, 0, 0), pw0 = pv0, pv1 = pv0, pw1 = pv0;
    if (b0 >= 0) { pv0 = w.pv_v[b0]; pw0 = w.pv_w[b0]; }
    if (b1 >= 0) { pv1 = w.pv_v[b1]; pw1 = w.pv_w[b1]; }
    joint_rows_presolve(w, q, pv0, pw0, pv1, pw1);
    if (b0 >= 0) { w.pv_v[b0] = pv0; w.pv_w[b0] = pw0; }
    if (b1 >= 0) { w.pv_v[b1] = pv1; w.pv_w[b1] = pw1; }
}

// The dynamic shared memory of the solver kernels: velocities, then contact records.
extern __shared__ float4 smem[];

// Body velocities the iterations work on, by scene-local dynamic body:
//   - SmemVel: in this block's shared memory, 24 bytes a body from its start, read and
//     written as three 8-byte words;
//   - ClusterVel: spread over the blocks of a thread-block cluster through distributed
//     shared memory (body i at block i mod 2^lg, index i >> lg), six float arrays of n;
//   - GlobVel: an array of the world (vt; in solve_flow also sv) from the scene's first body on.
// Each view is its own type so that every access has one known address space.
struct SmemVel {
    __device__ __forceinline__ void ld(int i, V3& v, V3& w) const {
        const float2* p = (const float2*)smem + 3 * i;
        const float2 a = p[0], b = p[1], c = p[2];
        v = {a.x, a.y, b.x};
        w = {b.y, c.x, c.y};
    }
    __device__ __forceinline__ void st(int i, V3 v, V3 w) const {
        float2* p = (float2*)smem + 3 * i;
        p[0] = make_float2(v.x, v.y);
        p[1] = make_float2(v.z, w.x);
        p[2] = make_float2(w.y, w.z);
    }
};
struct ClusterVel {
    float* const* rs;
    int n, lg;
    __device__ __forceinline__ void ld(int i, V3& v, V3& w) const {
        const float* b = rs[i & ((1 << lg) - 1)] + (i >> lg);
        v = {b[0], b[n], b[2 * n]};
        w = {b[3 * n], b[4 * n], b[5 * n]};
    }
    __device__ __forceinline__ void st(int i, V3 v, V3 w) const {
        float* b = rs[i & ((1 << lg) - 1)] + (i >> lg);
        b[0] = v.x; b[n] = v.y; b[2 * n] = v.z;
        b[3 * n] = w.x; b[4 * n] = w.y; b[5 * n] = w.z;
    }
};
struct GlobVel {
    float4* p;
    __device__ __forceinline__ void ld(int i, V3& v, V3& w) const { v = ld3(p[2 * i]); w = ld3(p[2 * i + 1]); }
    __device__ __forceinline__ void st(int i, V3 v, V3 w) const { p[2 * i] = st4(v); p[2 * i + 1] = st4(w); }
};
// Constraint1D(W)::solve for one row (Constraint1D.cpp:54-127 / Constraint1DW.cpp:117-233).
// V0, W0, V1, W1: the velocities of the joint's bodies (zero, and left so, for a side that
// is not simulated; both sides may be one body).  total: the row's accumulated
// impulse.  bias: 0.2 / h, formed once per substep (the device divides f64 slowly).
struct RowVals { float4 linear, angular0, angular1, angular0t, angular1t, misc; };
__device__ __forceinline__ void row_solve(const RowVals& r, float& total, float h, float bias, bool warm, const JointRun& J,
                                          V3& V0, V3& W0, V3& V1, V3& W1) {
    const bool simd = (J.rows >> 8) != 0, s0 = J.b0 >= 0, s1 = J.b1 >= 0, same = s0 && J.b0 == J.b1;
    const int fl = __float_as_int(r.angular0t.w);
    const bool angf = fl & 2, soft = fl & 1, lim = fl & 4;
    const float inv = r.angular1t.w;
    if (!simd && !inv) return;
    V3 v0 = V0, w0 = W0, v1 = V1, w1 = W1;
    const V3 l = ld3(r.linear), l0t = J.im0 * l, l1t = J.im1 * l, a0t = ld3(r.angular0t), a1t = ld3(r.angular1t);
    const float c = r.angular0.w;
    if (!soft && warm) {
        const bool apply = simd ? (fabsf(c) < (float)1e-4 && fabsf(total) < 10000.f)
                                : !((double)fabsf(c) > 1e-4 || fabsf(total) > 10000.f);
        if (apply) {
            const float lw = total * 0.5f;
            total = lw;
            if (!angf) { v0 += lw * l0t; v1 -= lw * l1t; }
            w0 += lw * a0t;
            w1 -= lw * a1t;
        }
    }
    if (simd && !inv) return;
    const V3 a0 = ld3(r.angular0), a1 = ld3(r.angular1);
    float rv = dot(a1, w1) - dot(a0, w0);
    if (!angf) rv += dot(l, v1) - dot(l, v0);
    const float tvel = r.linear.w, mn = r.angular1.w, mx = r.misc.x, freq = r.misc.y, damp = r.misc.z;
    float lambda;
    if (simd) {
        const float eff = 1.f / inv;
        if (soft) {
            float af = (2.f * kPi) * freq;
            float stiffness = af * af * eff;
            float damping = 2.f * af * damp * eff;
            float gamma = 1.f / (damping + h * stiffness);
            float beta = h * stiffness * gamma;
            lambda = (rv + beta * c / h) / (inv + gamma / h);
        } else {
            lambda = (rv - tvel + bias * c) * eff;
        }
    } else {
        if (soft) {
            float af = 2.f * kPi * freq;
            float stiffness = af * af / inv;
            float damping = 2.f * af * damp / inv;
            float gamma = 1.f / (damping + h * stiffness);
            float beta = h * stiffness / (damping + h * stiffness);
            lambda = (rv + beta * c / h) / (inv + gamma / h);
        } else {
            lambda = (rv - tvel + 0.2f * c / h) / inv;
        }
    }
    if (lim) {
        const float prev = total;
        total += lambda;
        if (simd) {
            float lo = mn * h, hi = mx * h;
            total = total > lo ? total : lo;
            total = total < hi ? total : hi;
        } else {
            total = clampG(total, mn, mx);
        }
        lambda = total - prev;
    } else {
        total += lambda;
    }
    // the scalar row applies only this iteration's impulse (Constraint1D.cpp:158-168): to
    // the stored velocities, not to those the warm start changed
    if (!simd) { v0 = V0; w0 = W0; }
    if (!angf) v0 += lambda * l0t;
    w0 += lambda * a0t;
    if (s0) { V0 = v0; W0 = w0; }
    if (!simd) {
        if (same) { V1 = V0; W1 = W0; }
        v1 = V1; w1 = W1;
    }
    if (!angf) v1 -= lambda * l1t;
    w1 -= lambda * a1t;
    if (s1) { V1 = v1; W1 = w1; }
    if (same) { V0 = V1; W0 = W1; }
}

// A joint's rows in solve order, on its bodies' velocities in registers; the next row's
// record is read while one is solved (a row is a chain of about twenty dependent
// operations, its record comes from L2).
__device__ __forceinline__ void joint_rows_solve(const World& w, int q, const JointRun& J, float h, float bias, bool warm,
                                                 V3& v0, V3& w0, V3& v1, V3& w1) {
    float4* R = joint_rows(w, q);
    const int n = J.rows & 0xff;
    auto read = [](const float4* r) {
        return RowVals{r[32 * ROW_LINEAR], r[32 * ROW_ANGULAR0], r[32 * ROW_ANGULAR1], r[32 * ROW_ANGULAR0T],
                       r[32 * ROW_ANGULAR1T], r[32 * ROW_MISC]};
    };
    if (!n) return;
    RowVals next = read(R);
    for (int i = 0; i < n; ++i, R += kRowStep) {
        const RowVals r = next;
        if (i + 1 < n) next = read(R + kRowStep);
        float total = r.misc.w;
        row_solve(r, total, h, bias, warm, J, v0, w0, v1, w1);
        R[32 * ROW_MISC].w = total;
    }
}

template <class V>
__device__ void joint_solve(const World& w, int q, float h, float bias, bool warm, int ds, const V vr) {
    const JointRun J = w.jruns[q];
    V3 v0 = {0, 0, 0}, w0 = {0, 0, 0}, v1 = {0, 0, 0}, w1 = {0, 0, 0};
    if (J.b0 >= 0) vr.ld(J.b0 - ds, v0, w0);
    if (J.b1 >= 0) vr.ld(J.b1 - ds, v1, w1);
    joint_rows_solve(w, q, J, h, bias, warm, v0, w0, v1, w1);
    if (J.b0 >= 0) vr.st(J.b0 - ds, v0, w0);
    if (J.b1 >= 0) vr.st(J.b1 - ds, v1, w1);
}

// ---------------------------------------------------------------- contacts (ContactConstraints.cpp)

__device__ __forceinline__ M3 world_invI(const World& w, int d) {
    return m3cols(ld3(w.mt[3 * d]), ld3(w.mt[3 * d + 1]), ld3(w.mt[3 * d + 2]));
}


// The constants of a contact's solver header.
__device__ void contact_header(const World& w, const Contact& c, int ds, int slots, SHdr& H) {
    H.n = c.n;
    H.m = make_float4(c.b0 >= 0 ? w.com[c.b0].w : 0.f, c.b1 >= 0 ? w.com[c.b1].w : 0.f, c.frequency, c.damping);
    H.i = make_int4(c.b0 >= 0 ? c.b0 - ds : -1, c.b1 >= 0 ? c.b1 - ds : -1, c.np | (c.soft ? HDR_SOFT : 0) | (slot_step(slots) << HDR_STEP), slot_first(slots));
}

// A contact's rows for one substep: the row update (src/Physecs.cpp:366-427), which reads
// the velocities the substep started with (w.vel, w.ang), then ContactConstraints::preSolve
// (src/ContactConstraints.cpp:4-31) and the per-substep constants of solve (:33-101), which
// read the integrated ones (vr).  `last`: the substep's separations stay with the contact.
template <class V>
__device__ void contact_rows(const World& w, Contact& c, SHdr& H, SPt* __restrict__ P, float h, bool last, const V vr) {
    const int4 id = *reinterpret_cast<const int4*>(&c.b0);   // b0, b1, body0, body1
    const int b0 = id.x, b1 = id.y, np = H.i.z & 0xff, step = H.i.z >> HDR_STEP;
    const bool soft = (H.i.z & HDR_SOFT) != 0;
    const float im0 = H.m.x, im1 = H.m.y;
    V3 com0 = {0, 0, 0}, v0 = {0, 0, 0}, w0 = {0, 0, 0}, com1 = {0, 0, 0}, v1 = {0, 0, 0}, w1 = {0, 0, 0};
    V3 nv0 = {0, 0, 0}, nw0 = {0, 0, 0}, nv1 = {0, 0, 0}, nw1 = {0, 0, 0};
    M3 I0 = m3zero(), I1 = m3zero();
    Q4 q0, q1;
    if (b0 >= 0) {
        com0 = ld3(w.bq[2 * b0]); q0 = ld4(w.bq[2 * b0 + 1]);
        v0 = ld3(w.vel[b0]); w0 = ld3(w.ang[b0]);
        I0 = world_invI(w, b0);
        vr.ld(H.i.x, nv0, nw0);
    } else q0 = ld4(w.quat[id.z]);
    if (b1 >= 0) {
        com1 = ld3(w.bq[2 * b1]); q1 = ld4(w.bq[2 * b1 + 1]);
        v1 = ld3(w.vel[b1]); w1 = ld3(w.ang[b1]);
        I1 = world_invI(w, b1);
        vr.ld(H.i.y, nv1, nw1);
    } else q1 = ld4(w.quat[id.w]);
    const V3 n = ld3(H.n);
    bool whole = np == 4;   // every row of the widest form is live
    for (int k = 0; k < np; ++k) {
        const float4 l0 = c.p[k].r0;
        const V3 r0 = qrot(q0, ld3(l0)), r1 = qrot(q1, ld3(c.p[k].r1));
        const V3 cp0 = com0 + r0, cp1 = com1 + r1;
        const float cc = dot(cp1 - cp0, n);
        const V3 rel = v1 + cross(w1, r1) - v0 - cross(w0, r0);
        const float relN = dot(rel, n);
        V3 t = rel - relN * n;
        const float tl = length(t);
        if (tl) t = t / tl;
        const V3 r0xn = cross(r0, n), r1xn = cross(r1, n), r0xt = cross(r0, t), r1xt = cross(r1, t);
        const V3 r0xnt = mv(I0, r0xn), r1xnt = mv(I1, r1xn), r0xtt = mv(I0, r0xt), r1xtt = mv(I1, r1xt);
        const float invN = dot(n, n) * (im0 + im1) + dot(r0xn, r0xnt) + dot(r1xn, r1xnt);
        const float invT = dot(t, t) * (im0 + im1) + dot(r0xt, r0xtt) + dot(r1xt, r1xtt);
        float t1 = 0.f, t2 = 0.f, lamT = 0.f;
        if (invN) {
            const float eff = 1.f / invN;
            if (soft) {
                const float af = 2.f * kPi * H.m.z;
                const float stiffness = af * af * eff;
                const float damping = 2.f * af * H.m.w * eff;
                const float gamma = 1.f / (damping + h * stiffness);
                const float beta = h * stiffness / (damping + h * stiffness);
                t1 = beta * cc / h;
                t2 = invN + gamma / h;
            } else {
                t1 = 0.1f * cc / h;
                t2 = eff;
            }
        }
        if (invT) {
            const float rv = dot(-t, nv0) + dot(-r0xt, nw0) + dot(t, nv1) + dot(r1xt, nw1);
            lamT = rv / invT;
        }
        const int live = (invN ? 1 : 0) | (invT ? 2 : 0);
        whole &= live == 3;
        SPt& p = P[k * step];
        p.a = make_float4(-r0xn.x, r1xn.x, -r0xn.y, r1xn.y);
        p.b = make_float4(-r0xn.z, r1xn.z, r0xnt.x, -r1xnt.x);
        p.c = make_float4(r0xnt.y, -r1xnt.y, r0xnt.z, -r1xnt.z);
        p.d = make_float4(0.f, l0.w, t1, t2);
        p.e = st4(t, 0.f);
        p.f = make_float4(r0xtt.x, -r1xtt.x, r0xtt.y, -r1xtt.y);
        p.g = make_float4(r0xtt.z, -r1xtt.z, lamT, __int_as_float(live));
        if (last) c.p[k].r1.w = cc;
    }
    // a -0 among the velocities; no sweep makes one that was not there (its bits are the least integer)
    auto least = [](const V3& a) { return min(min(__float_as_int(a.x), __float_as_int(a.y)), __float_as_int(a.z)); };
    const bool minus0 = !whole && min(min(least(nv0), least(nw0)), min(least(nv1), least(nw1))) == (int)0x80000000;
    if (minus0 != ((H.i.z & HDR_MINUS0) != 0)) H.i.z ^= HDR_MINUS0;
}

// Two floats in one 64-bit register; the packed operations round each lane as the scalar
// ones do, at half the instructions.  A packed product is formed as a * b + (-0), which is
// a * b exactly, with the -0 read from memory: the assembler contracts a packed multiply
// and the add that follows it into one fused operation, whatever its options.
struct F2 { unsigned long long u; };
__constant__ unsigned long long c_minus_zero2 = 0x8000000080000000ull;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2split(F2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.u)); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c_minus_zero2)); return r; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u)); return r; }
struct F2x3 { F2 x, y, z; };
__device__ __forceinline__ F2 dot(const F2x3& a, const F2x3& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// (a0, a1) += s * (b0, b1), each component
__device__ __forceinline__ void axpy(F2x3& a, F2 s, const F2x3& b) { a = {a.x + s * b.x, a.y + s * b.y, a.z + s * b.z}; }

// ContactConstraints::solve (src/ContactConstraints.cpp:33-124) of a contact with at most
// N points; ANY: the contact may be soft or hold a -0 (below).  No other thread touches the contact's bodies
// within its colour, so their velocities stay in registers from the first point to the
// last; every value equals a reload after each point.
// The step is one dependent chain of up to 2 N rows, so it is written for latency and
// few instructions:
//   * both bodies' sides of a row run as one packed operation (body 0, body 1), on
//     records that hold the two sides in pairs with the constraint's signs;
//   * the records are read ahead of the chain (the normal rows' all at once, then the
//     friction rows') and the accumulated impulses are written after the last row;
//   * all N rows of each kind are evaluated, with an impulse of zero where a row is not
//     live (the reference skips a row whose inverse effective mass is zero; a contact may
//     have fewer than N points) or a side has no simulated body, so the chain has no
//     branches.  A live row's operations and their order are the reference's (x - l * n
//     is formed as x + l * (-n), which rounds the same).  Adding a row of zeros changes
//     one value, a -0 to +0, so a contact that starts the substep with a -0 among its
//     velocities (HDR_MINUS0) takes the form that branches around rows that are not live.
//     (Selects there took registers from every form: 2.4 % of a frame of 2000 bodies; the
//     branches nothing.)
struct PairVel { V3 v0, w0, v1, w1; };   // a contact's or joint's velocities; zero on a side that is not simulated
template <int N, bool ANY>
__device__ __forceinline__ bool contact_solve(const SHdr& H, SPt* __restrict__ P, bool useBias, PairVel& pv) {
    const float friction = H.n.w;
    const int np = H.i.z & 0xff, step = H.i.z >> HDR_STEP;
    const bool soft = ANY && (H.i.z & HDR_SOFT) != 0;
    const bool sim0 = H.i.x >= 0, sim1 = H.i.y >= 0;
    const F2 im = f2(H.m.x, H.m.y);
    const F2x3 nm = {f2(-H.n.x, H.n.x), f2(-H.n.y, H.n.y), f2(-H.n.z, H.n.z)};
    const F2x3 np3 = {f2(H.n.x, -H.n.x), f2(H.n.y, -H.n.y), f2(H.n.z, -H.n.z)};
    // linear and angular velocities (body 0, body 1)
    F2x3 v = {f2(pv.v0.x, pv.v1.x), f2(pv.v0.y, pv.v1.y), f2(pv.v0.z, pv.v1.z)};
    F2x3 o = {f2(pv.w0.x, pv.w1.x), f2(pv.w0.y, pv.w1.y), f2(pv.w0.z, pv.w1.z)};
    // every normal record of the contact is read before the chain; rows past the
    // contact's points read its first point and stay dead
    float4 A[N], B[N], C[N], D[N];
    int live[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool has = i < np;
        const SPt* q = P + (has ? i * step : 0);
        A[i] = q->a; B[i] = q->b; C[i] = q->c; D[i] = q->d;
        live[i] = has ? __float_as_int(q->g.w) : 0;
    }
    bool touched = false;
    float lamN[N], lamT[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool on = (live[i] & 1) != 0;
        float lin0, lin1, ang0, ang1;
        f2split(dot(nm, v), lin0, lin1);
        f2split(dot(F2x3{f2(A[i].x, A[i].y), f2(A[i].z, A[i].w), f2(B[i].x, B[i].y)}, o), ang0, ang1);
        const float rv = lin0 + ang0 + lin1 + ang1;
        float lambda;
        if (soft) lambda = (rv + D[i].z) / D[i].w;
        else lambda = (rv - D[i].y + (useBias ? D[i].z : 0.f)) * D[i].w;
        const float prev = D[i].x;
        float tot = prev + lambda;
        tot = fminG(tot, 0.f);
        lamN[i] = on ? tot : prev;
        lambda = tot - prev;
        const F2 l = f2(on && sim0 ? lambda : 0.f, on && sim1 ? lambda : 0.f);
        if (!ANY || on) {
            axpy(v, l * im, np3);
            axpy(o, l, F2x3{f2(B[i].z, B[i].w), f2(C[i].x, C[i].y), f2(C[i].z, C[i].w)});
        }
        touched |= on;
    }
    float4 E[N], F[N], G[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int q = i < np ? i * step : 0;
        E[i] = P[q].e; F[i] = P[q].f; G[i] = P[q].g;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool on = (live[i] & 2) != 0;
        float lambda = G[i].z;
        const float limit = friction * lamN[i];
        const float prev = E[i].w;
        float tot = prev + lambda;
        tot = clampG(tot, limit, -limit);
        lamT[i] = tot;
        lambda = tot - prev;
        const F2 l = f2(on && sim0 ? lambda : 0.f, on && sim1 ? lambda : 0.f);
        if (!ANY || on) {
            axpy(v, l * im, F2x3{f2(E[i].x, -E[i].x), f2(E[i].y, -E[i].y), f2(E[i].z, -E[i].z)});
            axpy(o, l, F2x3{f2(F[i].x, F[i].y), f2(F[i].z, F[i].w), f2(G[i].x, G[i].y)});
        }
        touched |= on;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (live[i] & 1) P[i * step].d.x = lamN[i];
        if (live[i] & 2) P[i * step].e.w = lamT[i];
    }
    f2split(v.x, pv.v0.x, pv.v1.x); f2split(v.y, pv.v0.y, pv.v1.y); f2split(v.z, pv.v0.z, pv.v1.z);
    f2split(o.x, pv.w0.x, pv.w1.x); f2split(o.y, pv.w0.y, pv.w1.y); f2split(o.z, pv.w0.z, pv.w1.z);
    return touched;
}

// One contact of a colour step by the form that its warp needs: the contacts of a colour
// lie by point count (solve_scene), so a warp's contacts mostly have the same number, and
// most contacts of mixed shapes have one point (1.24 on average on the batched scenes).
// The vote only chooses among forms that all give this contact's result.
__device__ __forceinline__ bool contact_forms(const SHdr& H, SPt* __restrict__ P, bool useBias, PairVel& pv) {
    const int np = H.i.z & 0xff;
    const bool any = (H.i.z & (HDR_SOFT | HDR_MINUS0)) != 0;
    const unsigned lanes = __activemask();
    if (__any_sync(lanes, any)) return contact_solve<4, true>(H, P, useBias, pv);
    if (!__any_sync(lanes, np > 1)) return contact_solve<1, false>(H, P, useBias, pv);
    if (!__any_sync(lanes, np > 2)) return contact_solve<2, false>(H, P, useBias, pv);
    return contact_solve<4, false>(H, P, useBias, pv);
}

template <class V>
__device__ __forceinline__ void contact_step(const SHdr* __restrict__ Hp, SPt* __restrict__ points, bool useBias, const V vr) {
    const SHdr H = *Hp;
    if ((H.i.z & HDR_SOFT) && !useBias) return;   // the relaxation skips soft contacts
    const int b0 = H.i.x, b1 = H.i.y;
    PairVel pv = {};
    if (b0 >= 0) vr.ld(b0, pv.v0, pv.w0);
    if (b1 >= 0) vr.ld(b1, pv.v1, pv.w1);
    if (!contact_forms(H, points + H.i.w, useBias, pv)) return;
    if (b0 >= 0) vr.st(b0, pv.v0, pv.w0);
    if (b1 >= 0) vr.st(b1, pv.v1, pv.w1);
}

// ---------------------------------------------------------------- bodies

// integrate velocities (src/Physecs.cpp:441-469) into the solver's velocities; w.vel and
// w.ang keep the values the substep started with until its end.  Also stores what the
// contacts' rows read of the body.
template <bool FLOW, class V>
__device__ void integrate_velocity(const World& w, int d, int ds, float h, float g, const V vr) {
    int b = w.dyn_body[d];
    if (w.info[b].y & BODY_KIN) return;
    const Q4 q = ld4(w.quat[b]);
    w.bq[2 * d] = st4(ld3(w.pos[b]) + qrot(q, ld3(w.com[d])));
    w.bq[2 * d + 1] = st4(q);
    M3 rot = mat3_cast(q);
    M3 invRot = transpose(rot);
    V3 vel = ld3(w.vel[d]) + h * V3{0, -g, 0};
    V3 ang = ld3(w.ang[d]);
    V3 wl = mv(invRot, ang);
    M3 invIl = m3cols(ld3(w.invI[3 * d]), ld3(w.invI[3 * d + 1]), ld3(w.invI[3 * d + 2]));
    M3 I = inverse(invIl);
    V3 f = h * cross(wl, mv(I, wl));
    M3 J = madd(I, mscale(h, msub(mm(matrixCross3(wl), I), matrixCross3(mv(I, wl)))));
    wl = wl - solve33(J, f);
    ang = mv(rot, wl);
    vr.st(d - ds, vel, ang);
    if (FLOW) { w.sv[2 * d] = st4(vel); w.sv[2 * d + 1] = st4(ang); }
    w.pv_v[d] = make_float4(0, 0, 0, 0);
    w.pv_w[d] = make_float4(0, 0, 0, 0);
    M3 wi = mm(mm(rot, invIl), invRot);
    w.mt[3 * d] = st4(wi.c[0]);
    w.mt[3 * d + 1] = st4(wi.c[1]);
    w.mt[3 * d + 2] = st4(wi.c[2]);
}

// integrate positions (src/Physecs.cpp:492-512): lin, rot the solver's velocities of the
// body, pv and pw its pseudo velocities, `rows` the joint rows applied to them
__device__ __forceinline__ void integrate_position(const World& w, int d, int b, float h, V3 lin, V3 rot, V3 pv, V3 pw, float rows) {
    float s = rows != 0.f ? 1.f / rows : 1.f;
    V3 pos = ld3(w.pos[b]);
    Q4 q = ld4(w.quat[b]);
    V3 com = ld3(w.com[d]);
    pos += h * lin + s * pv;
    V3 prevCom = qrot(q, com);
    V3 wv = 0.5f * (h * rot + s * pw);
    q = qadd(q, qmul(Q4{wv.x, wv.y, wv.z, 0.f}, q));
    q = qnormalize(q);
    pos += prevCom - qrot(q, com);
    w.pos[b] = st4(pos);
    w.quat[b] = st4(q);
}

template <class V>
__device__ void integrate_position(const World& w, int d, int ds, float h, const V vr) {
    int b = w.dyn_body[d];
    if (w.info[b].y & BODY_KIN) return;
    const float4 pv = w.pv_v[d];
    V3 lin, rot;
    vr.ld(d - ds, lin, rot);
    integrate_position(w, d, b, h, lin, rot, ld3(pv), ld3(w.pv_w[d]), pv.w);
}

// ---------------------------------------------------------------- frame kernel

struct BlockSync {
    static constexpr bool kCluster = false, kBlock = true;
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int nth() const { return blockDim.x; }
    __device__ __forceinline__ bool any(bool v, int) const { return __syncthreads_or(v) != 0; }
    // block-wide maximum of v (v >= -1)
    __device__ int max_int(int v) const {
        __shared__ int mx;
        if (threadIdx.x == 0) mx = -1;
        __syncthreads();
        atomicMax(&mx, v);
        __syncthreads();
        int r = mx;
        __syncthreads();
        return r;
    }
};
struct GridSync {
    static constexpr bool kCluster = false, kBlock = false;
    GridBarrier bar;
    int* flag;
    __device__ __forceinline__ void sync() const { bar.sync(); }
    __device__ __forceinline__ int tid() const { return blockIdx.x * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ int nth() const { return gridDim.x * blockDim.x; }
    // Whether any thread of the grid holds v; `round` counts the calls, with a barrier between
    // two of them.  Three words take turns: this round's was cleared a round ago, and the one
    // that the round after the next uses, which every block has read by now, is cleared here.
    __device__ __forceinline__ bool any(bool v, int round) const {
        int* slot = flag + 2;
        if (threadIdx.x == 0 && blockIdx.x == 0) *(volatile int*)(slot + (round + 2) % 3) = 0;
        if (__syncthreads_or(v) && threadIdx.x == 0) atomicOr(slot + round % 3, 1);
        bar.sync();
        return *(volatile int*)(slot + round % 3) != 0;
    }
    // grid-wide maximum of v (v >= -1), through the barrier's spare word
    __device__ int max_int(int v) const {
        int* slot = flag + 1;
        if (threadIdx.x == 0 && blockIdx.x == 0) atomicExch(slot, -1);
        bar.sync();
        v = __reduce_max_sync(~0u, v);
        if ((threadIdx.x & 31) == 0) atomicMax(slot, v);
        bar.sync();
        int r = *(volatile int*)slot;
        bar.sync();
        return r;
    }
};

// A thread-block cluster working on one scene: the hardware cluster barrier orders
// shared, distributed-shared and global memory for all its threads; reductions go
// through a small array in block 0's shared memory.
struct ClusterSync {
    static constexpr bool kCluster = true, kBlock = false;
    int rank, R, lg;
    float* const* bases;   // every block's dynamic shared memory, mapped
    int* red;              // R ints in block 0's shared memory, mapped
    __device__ __forceinline__ void sync() const { cooperative_groups::this_cluster().sync(); }
    __device__ __forceinline__ int tid() const { return rank * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ int nth() const { return R * blockDim.x; }
    __device__ bool any(bool v, int) const {
        const int b = __syncthreads_or(v);
        if (threadIdx.x == 0) red[rank] = b;
        sync();
        int r = 0;
        for (int i = 0; i < R; ++i) r |= red[i];
        sync();
        return r != 0;
    }
    __device__ int max_int(int v) const {
        __shared__ int bm;
        if (threadIdx.x == 0) bm = -1;
        __syncthreads();
        atomicMax(&bm, v);
        __syncthreads();
        if (threadIdx.x == 0) red[rank] = bm;
        sync();
        int r = -1;
        for (int i = 0; i < R; ++i) r = max(r, red[i]);
        sync();
        return r;
    }
};

// Colouring of one scene's contacts (see solve_scene): first fit, in rounds.  Every
// uncoloured contact proposes the lowest colour that neither of its dynamic bodies
// carries yet (a 128-bit mask per body); each body accepts the lowest proposal, ties
// going to a hashed priority of the contact's index within the scene; a contact
// accepted by both bodies takes its colour.  At most one contact per body is coloured
// per round, so no two contacts of a colour share a dynamic body, and the result does
// not depend on thread timing.  mask[d - ds], claim[d - ds] (two sets of nd, taken in
// turn, so that one is reset while the other is in use), cb[k], col[k] are indexed
// by scene-local dynamic body and contact.  Contacts that find no colour below
// kMaxColors - 1 (bodies only gain colours, so such a contact never finds one) form a last
// colour that one thread solves in contact order; the return value is then negative.
//
// A round is two barriers and, but for the last, colours at least one contact: the lowest
// proposal of a round wins both its bodies.
template <class S>
__device__ int colour_contacts(const World& w, FrameBuf& f, int ms, int nc, int ds, int nd, const S& sy,
                               unsigned long long* claims, uint4* mask, int2* cb, int* col) {
    const int tid = sy.tid(), nth = sy.nth();
    const unsigned long long kFree = ~0ull;
    for (int d = tid; d < nd; d += nth) { claims[d] = kFree; mask[d] = make_uint4(0, 0, 0, 0); }
    for (int k = tid; k < nc; k += nth) {
        const int2 b = *reinterpret_cast<const int2*>(&f.contacts[ms + k].b0);
        const int2 l = make_int2(b.x >= 0 ? b.x - ds : -1, b.y >= 0 ? b.y - ds : -1);
        cb[k] = l;
        col[k] = l.x < 0 && l.y < 0 ? 0 : -1;
    }
    sy.sync();
    for (int round = 0;; ++round) {
        unsigned long long* claim = claims + (size_t)(round & 1) * nd;
        unsigned long long* other = claims + (size_t)(~round & 1) * nd;
        for (int d = tid; d < nd; d += nth) other[d] = kFree;
        for (int k = tid; k < nc; k += nth) {
            if (col[k] != -1) continue;
            const int2 b = cb[k];
            uint4 m0 = b.x >= 0 ? mask[b.x] : make_uint4(0, 0, 0, 0);
            uint4 m1 = b.y >= 0 ? mask[b.y] : make_uint4(0, 0, 0, 0);
            unsigned u[4] = {m0.x | m1.x, m0.y | m1.y, m0.z | m1.z, m0.w | m1.w};
            int c = kMaxColors - 1;
            for (int q = 0; q < 4; ++q)
                if (~u[q]) { c = 32 * q + __ffs(~u[q]) - 1; break; }
            if (c >= kMaxColors - 1) { col[k] = -2; continue; }   // no colour left: the serial colour takes it
            const unsigned long long v = claim_word(c, cache_hash((unsigned long long)k * 0x9E3779B97F4A7C15ull + round), k);
            if (b.x >= 0) atomicMin(&claim[b.x], v);
            if (b.y >= 0) atomicMin(&claim[b.y], v);
        }
        sy.sync();
        bool left = false;
        for (int k = tid; k < nc; k += nth) {
            if (col[k] != -1) continue;
            const int2 b = cb[k];
            const unsigned long long v0 = b.x >= 0 ? claim[b.x] : kFree, v1 = b.y >= 0 ? claim[b.y] : kFree;
            const bool mine0 = b.x < 0 || claim_of(v0, k);
            const bool mine1 = b.y < 0 || claim_of(v1, k);
            if (mine0 && mine1) {
                int c = claim_colour(b.x >= 0 ? v0 : v1);
                col[k] = c;
                // each body accepted only this contact this round: plain updates suffice
                unsigned bit = 1u << (c & 31);
                int q = c >> 5;
                if (b.x >= 0) { unsigned* mm = (unsigned*)&mask[b.x]; mm[q] |= bit; }
                if (b.y >= 0) { unsigned* mm = (unsigned*)&mask[b.y]; mm[q] |= bit; }
            } else {
                left = true;
            }
        }
        if (!sy.any(left, round)) break;
    }
    // colours used; contacts left without one form a last colour, solved serially
    int top = -1;
    for (int k = tid; k < nc; k += nth) top = max(top, col[k] < 0 ? kMaxColors : col[k]);
    top = sy.max_int(top);
    if (top < kMaxColors) return top + 1;
    // a contact without a colour means a body that carries all of them
    for (int k = tid; k < nc; k += nth) if (col[k] < 0) col[k] = kMaxColors - 1;
    sy.sync();
    return -kMaxColors;
}

// A scene's contacts in solve order: its first manifold, contacts, point slots, colours,
// whether the last colour is serial, and each colour's first contact.
struct SortedContacts {
    int ms, ncl, npts, ncol;
    bool serial_last;
    const int* colstart;
};

// All substeps of one scene.  SREC: contact records in shared memory (smem) from rec_f4 to
// smem_f4 as far as they fit, header and points of a contact together, from the last contact
// in solve order back to contact kg; the ones before keep theirs in the world's buffers.  A
// colour step with records in the world's buffers waits for them (some 4500 cycles against
// 1200 on 2000 mixed bodies), however few they are, and the first colour holds the most
// contacts: filled from the last, the others are all in shared memory (an iteration of that
// scene 12.0 -> 9.0 us).
template <bool SREC, class S, class V>
__device__ void solve_substeps(const World& w, FrameBuf& f, int s, const S& sy, const SortedContacts sc, int rec_f4,
                               int smem_f4, const V vr) {
    const int tid = sy.tid(), nth = sy.nth();
    const int ds = w.scene_dyn[s], de = w.scene_dyn[s + 1];
    const int ms = sc.ms, ncl = sc.ncl, ncol = sc.ncol;
    const float4 kn = w.knobs[s];
    const int substeps = (int)kn.x, iterations = (int)kn.y;
    const float g = kn.z, h = kn.w / substeps;
    int kg = ncl, slot0 = 0;   // the first contact in shared memory, and the first point slot there
    if constexpr (SREC) {
        const int room = smem_f4 - rec_f4;
        if (kHdrF4 * ncl + kPtF4 * sc.npts <= room) {
            kg = 0;
        } else {
            int fit = 0;
            for (int k = tid; k < ncl; k += nth)
                if (kHdrF4 * (ncl - k) + kPtF4 * (sc.npts - f.pt_group[ms + k]) <= room) fit = max(fit, ncl - k);
            kg = ncl - sy.max_int(fit);
            if (kg < ncl) slot0 = f.pt_group[ms + kg];
        }
    }
    // shared records: headers of contacts kg.., then point slots slot0.. (indexed as in the world's buffers)
    const int hdr_f4 = rec_f4 - kHdrF4 * kg, pts_f4 = rec_f4 + kHdrF4 * (ncl - kg) - kPtF4 * slot0;
    SHdr* const Hg = f.s_hdr + ms;
    SPt* const Pg = f.s_pts + 4 * (size_t)ms;
    auto HK = [&](int k) -> SHdr& { return SREC && k >= kg ? *(SHdr*)(smem + hdr_f4 + kHdrF4 * k) : Hg[k]; };
    auto PK = [&](int k) -> SPt* { return SREC && k >= kg ? (SPt*)(smem + pts_f4) : Pg; };
    for (int k = tid; k < ncl; k += nth) contact_header(w, f.contacts[f.corder[ms + k]], ds, f.pt_off[ms + k], HK(k));
    sy.sync();
    const int js0 = w.scene_jsteps[s], js1 = w.scene_jsteps[s + 1];
    const int jb = w.scene_joint[s], je = w.scene_joint[s + 1];   // schedule entries: every joint of the scene once
    const float joint_bias = jb < je ? (float)(0.2 / (double)h) : 0.f;
    for (int sub = 0; sub < substeps; ++sub) {
        for (int q = jb + tid; q < je; q += nth) make_joint_rows(w, q);
        for (int d = ds + tid; d < de; d += nth) integrate_velocity<false>(w, d, ds, h, g, vr);
        sy.sync();
        for (int k = tid; k < ncl; k += nth) {
            SHdr& H = HK(k);
            contact_rows(w, f.contacts[f.corder[ms + k]], H, PK(k) + H.i.w, h, sub == substeps - 1, vr);
        }
        for (int st = js0; st < js1; ++st) {
            for (int k = w.jstep_start[st] + tid; k < w.jstep_start[st + 1]; k += nth) joint_presolve(w, k);
            sy.sync();
        }
        sy.sync();
        // the iterations, then the positions and the relaxation (the sweep without bias)
        for (int it = 0; it <= iterations; ++it) {
            const bool bias = it < iterations;
            if (!bias) {
                for (int d = ds + tid; d < de; d += nth) integrate_position(w, d, ds, h, vr);
                sy.sync();
            }
            for (int cl = 0; cl < ncol; ++cl) {
                const bool serial = sc.serial_last && cl == ncol - 1;
                const int k1 = sc.colstart[cl + 1], stride = serial ? 1 : nth;
                int k = sc.colstart[cl] + tid;
                if (serial && tid != 0) k = k1;
                for (const int kw = SREC ? min(k1, kg) : k1; k < kw; k += stride) contact_step(Hg + k, Pg, bias, vr);
                if constexpr (SREC)
                    for (; k < k1; k += stride)
                        contact_step((const SHdr*)(smem + hdr_f4 + kHdrF4 * k), (SPt*)(smem + pts_f4), bias, vr);
                sy.sync();
            }
            if (bias)
                for (int st = js0; st < js1; ++st) {
                    for (int k = w.jstep_start[st] + tid; k < w.jstep_start[st + 1]; k += nth)
                        joint_solve(w, k, h, joint_bias, it == 0, ds, vr);
                    sy.sync();
                }
        }
        for (int d = ds + tid; d < de; d += nth) {
            int b = w.dyn_body[d];
            if (w.info[b].y & BODY_KIN) continue;
            V3 lin, rot;
            vr.ld(d - ds, lin, rot);
            w.vel[d] = st4(lin);
            w.ang[d] = st4(rot);
        }
        sy.sync();
    }
    // accumulated impulses back into the frame's contacts (inspection only)
    for (int k = tid; k < ncl; k += nth) {
        Contact& c = f.contacts[f.corder[ms + k]];
        const SHdr& H = HK(k);
        const SPt* q = PK(k) + H.i.w;
        const int step = H.i.z >> HDR_STEP;
        for (int i = 0; i < c.np; ++i) c.lambda[i] = make_float2(q[i * step].d.x, q[i * step].e.w);
    }
}

// ---- A scene solved by the whole grid without barriers between its colours.
//
// A sweep's order matters only body by body: a contact or joint may be solved as soon as the
// solves before it on its two bodies are done, and it touches nothing else.  So each body
// counts its solves of the substep in the w lanes of its velocities, every solve knows the
// counts it has to find (its place among its bodies' solves follows from the colours a
// body carries and from the joints' schedule), and a thread polls them, solves, and stores
// velocities and counts together.  The values are those of the sweep colour by colour.
// Each of a body's two 16-byte words is read and written whole and carries its count, so no
// fence is needed; records are only touched by the thread that solves them.
//
// A lane takes its solves in one order that is the same for all (sweep by sweep, contacts by
// colour, then joints by step), so the first open solve of the scene is always at the head
// of its lane's list and ready; all blocks are resident (cooperative launch).  The lanes of
// a warp poll together and none waits inside a divergent branch.
//
// A wait is bounded by what the grid does, not by its own length: a lane may rightly wait
// through every sweep of a substep (for the position of a body whose solves are other
// lanes'), and a block without work at the barrier after the last sweep, many times what a
// barrier after each colour waits.  So a wait whose polls reach the limit adds up the
// bodies' counts, and gives up only if none has moved since it last did so.
//
// Bound by the longest chain of solves on shared bodies, each a poll, a solve and a store
// through L2.  With a grid barrier after every colour and joint step, an iteration took
// 77.6 us on 65,536 bodies landing on a terrain (61,000 contacts in nine colours) and 104 us
// on 2048 chains of 32 links; so it takes 34.3 and 55.3 us (solver 3166 -> 1632 us and
// 4199 -> 2293 us a frame).
__device__ __forceinline__ void ld_stamped(const float4* p, V3& v, int& stamp) {
    unsigned long long a, b;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }" : "=l"(a), "=l"(b) : "l"(p));
    v = {__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)), __uint_as_float((unsigned)b)};
    stamp = (int)(b >> 32);
}
__device__ __forceinline__ void st_stamped(float4* p, V3 v, int stamp) {
    const unsigned long long a = __float_as_uint(v.x) | (unsigned long long)__float_as_uint(v.y) << 32;
    const unsigned long long b = __float_as_uint(v.z) | (unsigned long long)(unsigned)stamp << 32;
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p), "l"(a), "l"(b) : "memory");
}
// a body's two words, both at the count `want`
__device__ __forceinline__ bool ld_ready(const float4* p, int want, V3& v, V3& w, int& lag) {
    int s0, s1;
    ld_stamped(p, v, s0);
    ld_stamped(p + 1, w, s1);
    lag = max(lag, want - min(s0, s1));
    return s0 == want && s1 == want;
}

enum : int { FLOW_CONTACT, FLOW_JOINT, FLOW_POS, FLOW_OUT, FLOW_DONE };

__device__ void solve_flow(const World& w, FrameBuf& f, int s, const GridSync& sy, const SortedContacts sc) {
    // a warp's 32 solves lie next to each other; neighbouring warps of solves go to different blocks
    const int nth = sy.nth();
    const int slot = ((int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x) * 32 + (int)(threadIdx.x & 31);
    const int ds = w.scene_dyn[s], nd = w.scene_dyn[s + 1] - ds;
    const int ms = sc.ms, ncl = sc.ncl;
    const float4 kn = w.knobs[s];
    const int substeps = (int)kn.x, iterations = (int)kn.y;
    const float g = kn.z, h = kn.w / substeps;
    const int jq0 = w.scene_joint[s], jq1 = w.scene_joint[s + 1];   // schedule entries: every joint of the scene once
    const float joint_bias = jq0 < jq1 ? (float)(0.2 / (double)h) : 0.f;
    SHdr* const Hg = f.s_hdr + ms;
    SPt* const Pg = f.s_pts + 4 * (size_t)ms;
    float4* const vt = w.vt + 2 * (size_t)ds;
    auto carried = [&](int d, int below) {   // colours below `below` that body d carries
        const uint4 m = f.cmask[ds + d];
        const unsigned q[4] = {m.x, m.y, m.z, m.w};
        int n = 0;
        for (int i = 0; i < 4; ++i) {
            const int left = below - 32 * i;
            n += __popc(left >= 32 ? q[i] : (left <= 0 ? 0u : q[i] & ((1u << left) - 1u)));
        }
        return n;
    };
    for (int d = slot; d < nd; d += nth) {
        const int n = carried(d, kMaxColors);
        f.bdeg[ds + d] = flow_degree(n, w.body_nj[ds + d]);
    }
    for (int k = slot; k < ncl; k += nth) {
        SHdr& H = Hg[k];
        contact_header(w, f.contacts[f.corder[ms + k]], ds, f.pt_off[ms + k], H);
        const int c = f.color_of[f.corder[ms + k]];
        const int b0 = H.i.x, b1 = H.i.y;
        const int n0 = b0 >= 0 ? carried(b0, kMaxColors) + w.body_nj[ds + b0] : 0, r0 = b0 >= 0 ? carried(b0, c) : 0;
        const int n1 = b1 >= 0 ? carried(b1, kMaxColors) + w.body_nj[ds + b1] : 0, r1 = b1 >= 0 ? carried(b1, c) : 0;
        f.cbody[ms + k] = make_int2(r0 | n0 << 8, r1 | n1 << 8);   // place, and solves of the body per iteration
    }
    auto counts = [&](int first, int step) {   // of the bodies first, first + step, ...: solves and preSolves done
        unsigned all = 0;
        for (int d = first; d < nd; d += step)
            all += *(volatile unsigned*)&vt[2 * d].w + *(volatile unsigned*)&w.pv_w[ds + d].w;
        return all;
    };
    for (int sub = 0; sub < substeps; ++sub) {
        for (int q = jq0 + slot; q < jq1; q += nth) make_joint_rows(w, q);
        for (int d = slot; d < nd; d += nth) integrate_velocity<true>(w, ds + d, ds, h, g, GlobVel{vt});
        sy.sync();
        for (int k = slot; k < ncl; k += nth)
            contact_rows(w, f.contacts[f.corder[ms + k]], Hg[k], Pg + Hg[k].i.w, h, sub == substeps - 1,
                         GlobVel{w.sv + 2 * (size_t)ds});
        // the lane's current solve: in sweep `it` (-1: the joints' preSolve, `iterations`: the
        // positions, the relaxation and the result), its bodies and the counts it waits for
        int it = -1, kind = FLOW_JOINT, idx = jq0 + slot, b0 = -1, b1 = -1, e0 = 0, e1 = 0;
        int4 hi = make_int4(0, 0, 0, 0);
        auto settle = [&]() {   // on to the next solve that exists, from (it, kind, idx); then reads what it waits for
            while (true) {
                if (kind == FLOW_JOINT) {
                    if (idx < jq1) break;
                    ++it;
                    kind = it < iterations ? FLOW_CONTACT : FLOW_POS;
                    idx = slot;
                } else if (kind == FLOW_CONTACT) {
                    if (idx < ncl) break;
                    kind = it < iterations ? FLOW_JOINT : FLOW_OUT;
                    idx = it < iterations ? jq0 + slot : slot;
                } else if (kind == FLOW_POS || kind == FLOW_OUT) {
                    if (idx < nd) {
                        if (!(w.info[w.dyn_body[ds + idx]].y & BODY_KIN)) break;
                        idx += nth;
                    } else {
                        kind = kind == FLOW_POS ? FLOW_CONTACT : FLOW_DONE;
                        idx = slot;
                    }
                } else return;
            }
            if (kind == FLOW_CONTACT) {
                hi = Hg[idx].i;
                const int2 place = f.cbody[ms + idx];
                b0 = hi.x; b1 = hi.y;
                const int relax = it == iterations;   // after the position integration
                e0 = (place.x & 0xff) + it * (place.x >> 8) + relax;
                e1 = (place.y & 0xff) + it * (place.y >> 8) + relax;
            } else if (kind == FLOW_JOINT) {
                const JointRun J = w.jruns[idx];
                b0 = J.b0 >= 0 ? J.b0 - ds : -1;
                b1 = J.b1 >= 0 ? J.b1 - ds : -1;
                const int d0 = b0 >= 0 && it >= 0 ? f.bdeg[J.b0] : 0, d1 = b1 >= 0 && it >= 0 ? f.bdeg[J.b1] : 0;
                e0 = J.rank0 + flow_contacts(d0) + max(it, 0) * flow_solves(d0);
                e1 = J.rank1 + flow_contacts(d1) + max(it, 0) * flow_solves(d1);
            } else {
                const int deg = f.bdeg[ds + idx];
                b0 = idx; b1 = -1;
                e0 = iterations * flow_solves(deg) + (kind == FLOW_OUT ? 1 + flow_contacts(deg) : 0);
                e1 = w.body_nj[ds + idx];   // preSolves the position integration waits for
            }
        };
        settle();
        unsigned seen = 0;   // the counts when this warp last added them up
        for (long long polls = 0; __any_sync(~0u, kind != FLOW_DONE);) {
            PairVel pv = {};
            float4 ps0 = make_float4(0, 0, 0, 0), pw0 = ps0, ps1 = ps0, pw1 = ps0;
            bool ready = kind != FLOW_DONE;
            int lag = 0;
            if (kind == FLOW_DONE) {
            } else if (kind == FLOW_JOINT && it < 0) {
                // pseudo velocities: the rows applied so far with the preSolves done, and the latter
                auto ready_pseudo = [&](int b, int want, float4& a, float4& c) {
                    V3 x, y;
                    int s0, s1;
                    ld_stamped(w.pv_v + ds + b, x, s0);
                    ld_stamped(w.pv_w + ds + b, y, s1);
                    a = st4(x, (float)flow_pseudo_rows(s0));
                    c = st4(y, 0.f);
                    return flow_pseudo_joints(s0) == want && s1 == want;
                };
                if (b0 >= 0) ready &= ready_pseudo(b0, e0, ps0, pw0);
                if (b1 >= 0) ready &= ready_pseudo(b1, e1, ps1, pw1);
            } else {
                if (b0 >= 0) ready &= ld_ready(vt + 2 * b0, e0, pv.v0, pv.w0, lag);
                if (b1 >= 0) ready &= ld_ready(vt + 2 * b1, e1, pv.v1, pv.w1, lag);
                if (kind == FLOW_POS && ready) {
                    V3 x, y;
                    int s0, s1;
                    ld_stamped(w.pv_v + ds + b0, x, s0);
                    ld_stamped(w.pv_w + ds + b0, y, s1);
                    ready = flow_pseudo_joints(s0) == e1 && s1 == e1;
                    ps0 = st4(x, (float)flow_pseudo_rows(s0));
                    pw0 = st4(y);
                }
            }
            if (ready) {
                if (kind == FLOW_CONTACT) {
                    const bool bias = it < iterations;
                    if (bias || !(hi.z & HDR_SOFT)) contact_forms(Hg[idx], Pg + hi.w, bias, pv);
                } else if (kind == FLOW_JOINT) {
                    if (it < 0) joint_rows_presolve(w, idx, ps0, pw0, ps1, pw1);
                    else joint_rows_solve(w, idx, w.jruns[idx], h, joint_bias, it == 0, pv.v0, pv.w0, pv.v1, pv.w1);
                } else if (kind == FLOW_POS) {
                    integrate_position(w, ds + b0, w.dyn_body[ds + b0], h, pv.v0, pv.w0, ld3(ps0), ld3(pw0), ps0.w);
                } else {
                    w.vel[ds + b0] = st4(pv.v0);
                    w.ang[ds + b0] = st4(pv.w0);
                }
                if (kind == FLOW_JOINT && it < 0) {
                    if (b0 >= 0) { st_stamped(w.pv_v + ds + b0, ld3(ps0), flow_pseudo((int)ps0.w, e0 + 1)); st_stamped(w.pv_w + ds + b0, ld3(pw0), e0 + 1); }
                    if (b1 >= 0) { st_stamped(w.pv_v + ds + b1, ld3(ps1), flow_pseudo((int)ps1.w, e1 + 1)); st_stamped(w.pv_w + ds + b1, ld3(pw1), e1 + 1); }
                } else if (kind != FLOW_OUT) {
                    if (b0 >= 0) { st_stamped(vt + 2 * b0, pv.v0, e0 + 1); st_stamped(vt + 2 * b0 + 1, pv.w0, e0 + 1); }
                    if (b1 >= 0) { st_stamped(vt + 2 * b1, pv.v1, e1 + 1); st_stamped(vt + 2 * b1 + 1, pv.w1, e1 + 1); }
                }
                idx += nth;
                settle();
                polls = 0;
            } else if (kind != FLOW_DONE) {
                // a wait that ran out, here or elsewhere, ends the lane's list; the grid leaves at the next barrier
                if ((++polls & 63) == 0 && (*(volatile int*)w.err & ERR_BARRIER_TIMEOUT)) kind = FLOW_DONE;
            }
            if (!__any_sync(~0u, ready)) {
                // nothing to do yet: the further the nearest solve, the longer the pause (-1: a wait at its limit)
                const int near = __reduce_min_sync(~0u, kind == FLOW_DONE ? 1 << 20 : polls > sy.bar.limit ? -1 : lag);
                if (near < 0) {
                    const unsigned all = __reduce_add_sync(~0u, counts(slot & 31, 32));
                    if (all == seen && kind != FLOW_DONE && polls > sy.bar.limit) {
                        atomicOr(w.err, ERR_BARRIER_TIMEOUT);
                        kind = FLOW_DONE;
                    }
                    if (all != seen) polls = 0;
                    seen = all;
                }
                __nanosleep(near > 3 ? 400 : 40);
            }
        }
        sy.bar.sync([&] { return counts(0, 1); });
    }
    // accumulated impulses back into the frame's contacts (inspection only)
    for (int k = slot; k < ncl; k += nth) {
        Contact& c = f.contacts[f.corder[ms + k]];
        const SHdr& H = Hg[k];
        const SPt* q = Pg + H.i.w;
        const int step = H.i.z >> HDR_STEP;
        for (int i = 0; i < c.np; ++i) c.lambda[i] = make_float2(q[i * step].d.x, q[i * step].e.w);
    }
}

template <class S>
__device__ void solve_scene(const World& w, FrameBuf& f, int s, const S& sy, int smem_f4) {
    if (w.scene_active && !w.scene_active[s]) return;
    const int tid = sy.tid(), nth = sy.nth();
    int ds = w.scene_dyn[s], de = w.scene_dyn[s + 1];
    int ms = f.scene_man[s], me = f.scene_man[s + 1];
    // bins of the counting sort: bin_a counts, then cursors; bin_b as written by the scan
    __shared__ int bin_a[kColorBins], bin_b[kColorBins], bin_total[2];
    __shared__ int colstart[kMaxColors + 1];   // first contact of each colour, read by every colour step
    // ---- graph colouring of the contacts (colour_contacts).  Priorities use the contact's
    // index within its scene, so a scene is coloured the same way whatever other scenes
    // share the world.  The working arrays (bodies of each contact, colour of each
    // contact, two claim words per dynamic body) live in shared memory when they fit.
    const int nd = de - ds, nc = me - ms;
    const bool col_smem = !S::kCluster && 32 * (size_t)nd + 12 * (size_t)nc <= 16 * (size_t)smem_f4;
    uint4* cmask = col_smem ? (uint4*)smem : f.cmask + ds;
    unsigned long long* claim = col_smem ? (unsigned long long*)(cmask + nd) : f.claim + 2 * (size_t)ds;
    int2* cb = col_smem ? (int2*)(claim + 2 * nd) : f.cbody + ms;
    int* col = col_smem ? (int*)(cb + nc) : f.color_of + ms;
    int ncol = colour_contacts(w, f, ms, nc, ds, nd, sy, claim, cmask, cb, col);
    const bool serial_last = ncol < 0;
    if (serial_last) ncol = -ncol;
    // Counting sort of the scene's contacts by colour and, within a colour, by point count
    // (four points first), one bin each: contacts of one colour touch disjoint bodies and
    // may be solved in any order, and a warp of contacts with the same point count runs no
    // row it does not need.  A contact's point slots follow from its bin, so the records
    // are packed without a scan over the contacts.  A block keeps the bins in shared
    // memory, a grid or cluster counts in global memory and scans once per block.
    const int nbins = kPointBins * ncol;
    int* const hist = S::kBlock ? bin_a : f.color_start + (size_t)s * kColorBins;
    int* const cursor = S::kBlock ? bin_a : f.claim_pos + (size_t)s * kColorBins;
    auto bin_of = [&](int cl, int k) {
        if (serial_last && cl == ncol - 1) return kPointBins * cl;
        return kPointBins * cl + 4 - min(4, max(1, f.contacts[ms + k].np));
    };
    for (int b = tid; b < nbins; b += nth) { hist[b] = 0; if (!S::kBlock) cursor[b] = 0; }
    sy.sync();
    for (int k = tid; k < nc; k += nth) { const int cl = col[k]; if (cl >= 0) atomicAdd(&hist[bin_of(cl, k)], 1); }
    sy.sync();
    if (threadIdx.x < 32) {
        // bin_a: first contact of the bin; bin_b: its first point slot
        int c0 = 0, p0 = 0;
        for (int base = 0; base < nbins; base += 32) {
            const int b = base + (int)threadIdx.x, per = 4 - (b & (kPointBins - 1));
            const int n = b < nbins ? (S::kBlock ? bin_a[b] : ((volatile int*)hist)[b]) : 0;
            int cs = n, ps = n * per;
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(~0u, cs, o), y = __shfl_up_sync(~0u, ps, o);
                if ((int)threadIdx.x >= o) { cs += x; ps += y; }
            }
            if (b < nbins) {
                bin_a[b] = c0 + cs - n;
                bin_b[b] = p0 + ps - n * per;
            }
            c0 += __shfl_sync(~0u, cs, 31);
            p0 += __shfl_sync(~0u, ps, 31);
        }
        if (threadIdx.x == 0) { bin_total[0] = c0; bin_total[1] = p0; }
    }
    if (tid == 0) f.scene_ncolor[s] = ncol;
    __syncthreads();
    const int ncl = bin_total[0], npts = bin_total[1];   // coloured contacts (all of them) and their point slots
    for (int c = threadIdx.x; c <= ncol; c += blockDim.x) colstart[c] = c < ncol ? bin_a[kPointBins * c] : ncl;
    __syncthreads();
    for (int k = tid; k < nc; k += nth) {
        const int cl = col[k];
        if (S::kBlock) f.color_of[ms + k] = cl;   // kept for inspection
        if (cl < 0 || (serial_last && cl == ncol - 1)) continue;
        const int b = bin_of(cl, k);
        const int pos = atomicAdd(&cursor[b], 1) + (S::kBlock ? 0 : bin_a[b]);
        f.corder[ms + pos] = ms + k;
    }
    if (serial_last && tid == 0) {
        // the serial colour keeps contact order
        int pos = colstart[ncol - 1];
        for (int k = 0; k < nc; ++k)
            if (col[k] == ncol - 1) f.corder[ms + pos++] = ms + k;
    }
    sy.sync();
    // Point slots: eight contacts of a bin side by side (fewer at its end), point by point,
    // so that the lanes of a warp read a point of theirs at 112-byte steps, which hit every
    // bank once; a contact's points in a row (448 bytes a contact) put sixteen lanes on
    // four banks.  pt_off: the contact's first slot and the step between its points
    // (slot_word); pt_group: the first of its eight contacts' slots.
    for (int k = tid; k < ncl; k += nth) {
        const int m = f.corder[ms + k] - ms, b = bin_of(f.color_of[ms + m], m), per = 4 - (b & (kPointBins - 1));
        // in block mode the cursors have moved on to each bin's end
        const bool serial = serial_last && b == kPointBins * (ncol - 1);
        const int c0 = serial ? colstart[ncol - 1] : (S::kBlock ? (b ? bin_a[b - 1] : 0) : bin_a[b]);
        const int c1 = serial ? ncl : (S::kBlock ? bin_a[b] : (b + 1 < nbins ? bin_a[b + 1] : ncl));
        const int i = k - c0, t8 = i & ~7, step = min(8, c1 - c0 - t8);
        f.pt_off[ms + k] = slot_word(bin_b[b] + t8 * per + (i & 7), step);
        f.pt_group[ms + k] = bin_b[b] + t8 * per;
    }
    sy.sync();
    const SortedContacts sc{ms, ncl, npts, ncol, serial_last, colstart};
    const int vel_f4 = (6 * nd + 3) / 4;
    if constexpr (S::kBlock) {
        if (vel_f4 <= smem_f4) solve_substeps<true>(w, f, s, sy, sc, vel_f4, smem_f4, SmemVel{});
        else solve_substeps<false>(w, f, s, sy, sc, 0, 0, GlobVel{w.vt + 2 * (size_t)ds});
    } else if constexpr (S::kCluster) {
        // velocities spread over the cluster's blocks; records and colouring stay global
        const int per = (nd + sy.R - 1) >> sy.lg;
        if (6 * per <= 4 * smem_f4) solve_substeps<false>(w, f, s, sy, sc, 0, 0, ClusterVel{sy.bases, per, sy.lg});
        else solve_substeps<false>(w, f, s, sy, sc, 0, 0, GlobVel{w.vt + 2 * (size_t)ds});
    } else {
        // a colour beyond the limit is solved in contact order, which the counts do not express,
        // and a body of very many joints outgrows them
        if (serial_last || w.no_flow) solve_substeps<false>(w, f, s, sy, sc, 0, 0, GlobVel{w.vt + 2 * (size_t)ds});
        else solve_flow(w, f, s, sy, sc);
    }
}

// one scene per block; by size NT = 32 or 64, 128 or 256, and 512 for the world's large scenes: above
// 1024 dynamic bodies, or above 192 where no more scenes than SMs are (build_world)
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_solve_block(World w, FrameBuf f, const int* scenes, int smem_f4) {
    BlockSync sy;
    solve_scene(w, f, scenes[blockIdx.x], sy, smem_f4);
}

static_assert(kBarrierTimeoutBit == ERR_BARRIER_TIMEOUT, "grid barrier error bit");

__global__ void __launch_bounds__(256, 2) k_solve_grid(World w, FrameBuf f, const int* scenes, int n, long long limit) {
    GridSync sy{GridBarrier{f.bar, f.bar + 1, w.err, limit}, (int*)(f.bar + 2)};
    for (int i = 0; i < n; ++i) {
        solve_scene(w, f, scenes[i], sy, 0);
        sy.sync();
    }
}

// one cluster of kClusterBlocks blocks per large scene, velocities in distributed shared memory
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_solve_cluster(World w, FrameBuf f, const int* scenes, int smem_f4) {
    __shared__ float* bases[kClusterBlocks];
    __shared__ int red[kClusterBlocks];
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int R = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    if (threadIdx.x < R) bases[threadIdx.x] = cl.map_shared_rank((float*)smem, (int)threadIdx.x);
    int* red0 = cl.map_shared_rank(red, 0);
    int lg = 0;
    while ((1 << lg) < R) ++lg;
    cl.sync();
    ClusterSync sy{rank, R, lg, bases, red0};
    solve_scene(w, f, scenes[blockIdx.x / R], sy, smem_f4);
    cl.sync();   // no block leaves while the others may still read its shared memory
}

int launch_contacts(const World& w, FrameBuf& f, cudaStream_t s) {
    const int cells = std::max(f.cache_cap, w.n_scenes + 1);
    k_contacts_begin<<<(cells + 255) / 256, 256, 0, s>>>(f, w.n_scenes);
    k_build_contacts<<<1216, kContactThreads, 0, s>>>(w, f);
    return 2 + scan_exclusive(f.man_scene_cnt, f.scene_man, w.n_scenes + 1, nullptr, f.scan_scratch, s);
}

int solver_grid_blocks() {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_solve_grid, 256, 0);
    if (per < 1) per = 1;
    return sms * per;
}

static void set_kernel_smem(const void* fn, SmemLimit& limit, int bytes) {
    int dev = 0;
    cudaGetDevice(&dev);
    limit.raise(dev, bytes, [fn](int b) { cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, b); });
}

template <int NT>
static void set_smem(int bytes) {
    static SmemLimit limit;
    set_kernel_smem((const void*)k_solve_block<NT>, limit, bytes);
}

// A solver launch at a scheduling priority: `rank` 0 is the device's highest, each step
// one lower, down to the lowest (the priority is a launch attribute, so a CUDA graph
// captured from it keeps it).  The larger the scenes of a launch, the longer their
// chains and the earlier their blocks should start.
template <int NT>
static void launch_block_ranked(int grid, int smem, cudaStream_t st, int rank, const World& w, FrameBuf& f,
                                const int* scenes) {
    int least = 0, greatest = 0;
    cudaDeviceGetStreamPriorityRange(&least, &greatest);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = greatest < least ? std::min(least, greatest + rank) : greatest;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_solve_block<NT>, w, f, scenes, smem / 16);
}

int launch_solver(const World& w, FrameBuf& f, const SolverLaunch& L, cudaStream_t s) {
    int k = 0;
    // large scenes on a second stream, concurrently with the small ones, and first: their
    // chains are the longest (measured with eager launches: solver stage 7.20 -> 6.65 ms
    // on the 4096-scene frame)
    if (L.n_large) {
        cudaEventRecord(L.fork, s);
        cudaStreamWaitEvent(L.aux, L.fork, 0);
        if (L.large_nt == 128 || L.large_nt == 256) {
            // several blocks an SM, each with its share of the SM's shared memory (beside
            // each block's 1 KB reserve and its static shared memory)
            const int per = L.large_nt == 128 ? 4 : 2;
            const int smem = (L.smem_large + 5120 - per * 6144) / per / 16 * 16;
            if (L.large_nt == 128) {
                set_smem<128>(smem);
                launch_block_ranked<128>(L.n_large, smem, L.aux, 0, w, f, L.large);
            } else {
                set_smem<256>(smem);
                launch_block_ranked<256>(L.n_large, smem, L.aux, 0, w, f, L.large);
            }
        } else {
            set_smem<512>(L.smem_large);
            launch_block_ranked<512>(L.n_large, L.smem_large, L.aux, 0, w, f, L.large);
        }
        cudaEventRecord(L.join, L.aux);
        ++k;
    }
    // block scenes: 64- and 128-thread tiers on their own streams beside the 256-thread one
    if (L.n_tier[0] || L.n_tier[1]) cudaEventRecord(L.tfork, s);
    if (L.n_tier[0]) {
        cudaStreamWaitEvent(L.tstream[0], L.tfork, 0);
        if (L.tier0_nt == 32) {   // one warp a scene: up to 16 scenes an SM
            set_smem<32>(L.smem_tier[0]);
            launch_block_ranked<32>(L.n_tier[0], L.smem_tier[0], L.tstream[0], 3, w, f, L.tier[0]);
        } else {
            set_smem<64>(L.smem_tier[0]);
            launch_block_ranked<64>(L.n_tier[0], L.smem_tier[0], L.tstream[0], 3, w, f, L.tier[0]);
        }
        cudaEventRecord(L.tjoin[0], L.tstream[0]);
        ++k;
    }
    if (L.n_tier[1]) {
        set_smem<128>(L.smem_tier[1]);
        cudaStreamWaitEvent(L.tstream[1], L.tfork, 0);
        launch_block_ranked<128>(L.n_tier[1], L.smem_tier[1], L.tstream[1], 2, w, f, L.tier[1]);
        cudaEventRecord(L.tjoin[1], L.tstream[1]);
        ++k;
    }
    if (L.n_tier[2]) {
        set_smem<256>(L.smem_tier[2]);
        launch_block_ranked<256>(L.n_tier[2], L.smem_tier[2], s, 1, w, f, L.tier[2]);
        ++k;
    }
    if (L.n_tier[0]) cudaStreamWaitEvent(s, L.tjoin[0], 0);
    if (L.n_tier[1]) cudaStreamWaitEvent(s, L.tjoin[1], 0);
    if (L.n_large) cudaStreamWaitEvent(s, L.join, 0);
    if (L.n_cluster) {
        static SmemLimit cluster_smem;
        set_kernel_smem((const void*)k_solve_cluster<512>, cluster_smem, L.smem_large);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterBlocks * L.n_cluster);
        cfg.blockDim = dim3(512);
        cfg.dynamicSmemBytes = L.smem_large;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClusterBlocks;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k_solve_cluster<512>, w, f, L.cluster, L.smem_large / 16);
        ++k;
    }
    if (L.n_grid) {
        World wc = w;
        FrameBuf fc = f;
        const int* gs = L.grid;
        int ng = L.n_grid;
        long long limit = L.wait_limit > 0 ? L.wait_limit : kDefaultWaitPolls;
        // the barrier's words start from zero in every launch, whatever an earlier launch
        // that gave up on a wait left in them
        cudaMemsetAsync(f.bar, 0, kBarWords * sizeof(unsigned), s);
        void* args[] = {(void*)&wc, (void*)&fc, (void*)&gs, (void*)&ng, (void*)&limit};
        cudaLaunchCooperativeKernel((void*)k_solve_grid, L.grid_blocks, 256, args, 0, s);
        ++k;
    }
    return k;
}

}  // namespace psx
