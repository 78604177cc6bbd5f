// kernels.cuh -- sm_100a kernels of the B200 DEM engine.
//
// Step structure.  k_steps takes many steps in a launch, the graph's loop puts the
// rebuilds between its launches (engine.cu, capture_loop); timed, eager and
// export steps launch the passes one by one:
//   k_clump      per clump: member force/torque sum and second half-kick of
//                the previous step, first half-kick, drift, attitude and the
//                pose of every member subsphere (+ rebuild test); one extra
//                thread per scene advances the intruder.
//   [rebuild]    only when some scene's subsphere moved more than Thresh
//                since that scene's last rebuild: cell hash with counts,
//                counting sort (the reference's stable order) with the reorder,
//                half search into back rows, scans, back rows and the owners'
//                unordered front rows, front rows in order with the reverse
//                map, the contact pass's work records and carried histories
//   k_pairs      per near pair: overlap test, the law once for both
//                subspheres of a touching pair, the new spring history, the
//                force and torque on each side into its contact slot
//   k_boundary   per boundary candidate: walls and intruder (beside k_pairs)
//   (the next step's k_clump sums each member's slots and boundary force)
#pragma once
#include "nbc_dev.cuh"
#include "nbc_math.cuh"

namespace nbc {

constexpr double FIX_F = 1099511627776.0;    // 2^40: fixed-point scale of intruder force sums
constexpr double FIX_T = 17592186044416.0;   // 2^44: fixed-point scale of intruder torque sums
constexpr int IDX_MASK = 0x7fffffff;
constexpr int INTRA = (int)0x80000000u;

// ===========================================================================
// clump pass
// ===========================================================================

// Integrate_Before_clump_cuk / Attitude_clump_cuk / Integrate_After_clump_cuk
// (src/dem_integrate_clumpsphere.cu:3-141), UpdatePos_cuk (src/dem_clump.cu:
// 113-138), ComputeTorqueFromWorldPos_Kernel + reduce_by_key
// (src/dem_clumpsphere.cu:86-151), IntegratePene_Before_cuk and
// Integrate_After_cuk (src/dem_integrate_penetrator.cu:3-113).
//
// One member per lane.  The host packs whole clumps into warps (Dev::lrec, a
// record per lane; members of a clump are consecutive lanes, a clump of more
// than 32 members has a warp of its own that walks them 32 at a time, a clump
// without members one lane).  A lane sums its member's contact slots, forms
// the lever-arm torque, and the lanes of a clump add up their members in
// ascending order through shuffles (the reduce_by_key order); every lane then
// integrates its clump (a warp instruction costs the same for one lane as for
// 32), poses its own member from registers, and the clump's first lane writes
// the clump.  The warps after the last one of the table hold one thread per
// scene for the intruder.
//
// Bound by latency: a chain of four dependent loads (lane record, member
// index, row offsets and member records, slots), the FP64 integration, the
// stores.  One lane per clump, with the members of a warp's 32 clumps walked
// through shared memory in four or more chunks, put that chain in series four
// times and left 391 blocks of work for 50,000 clumps (events around the pass,
// one lane per clump -> one per member: 500 clumps 20.6 -> 12.4 us, 13,331 in
// FP64 27.2 -> 15.8, 50,000 32.8 -> 34.2, 250,000 141 -> 151).
//
// A step (do_pre) also advances the spring-history generation so the next
// contact pass reads what the previous one wrote, and counts itself; the last
// block to finish sets the graph's rebuild condition (when given a handle)
// and counts the step in lstep.  A scene with a stop s takes the steps started
// at lstep = 0 .. s-1 and closes the last one at lstep = s; afterwards it
// stands still (frozen) while the other scenes go on, so its state is
// exactly that of the scene run alone for s steps.
__device__ __forceinline__ bool scene_pre(const SceneDyn& y, int do_pre, int L) {
    return do_pre && (y.stop == 0 || L < y.stop);
}
__device__ __forceinline__ bool scene_post(const SceneDyn& y, int post, int L) {
    return post && (y.stop == 0 || L <= y.stop);
}
constexpr int CL_THREADS = 128;
constexpr int CL_WARPS = CL_THREADS / 32;
#ifndef NBC_CLUMP_MINB
#define NBC_CLUMP_MINB 4
#endif
// One attitude step (Attitude_clump_cuk, src/dem_integrate_clumpsphere.cu:45-90).
__device__ __forceinline__ double4 quat_step(double4 q, V3<double> w, V3<double> al, double Dt) {
    const V3<double> Wb = rot_w2b(q, w), Wdb = rot_w2b(q, al);
    double4 qd, qdd, r;
    qd.x = 0.50 * fma3(Wb.x, q.w, -Wb.y, q.z, Wb.z, q.y);
    qd.y = 0.50 * fma3(Wb.x, q.z, Wb.y, q.w, -Wb.z, q.x);
    qd.z = 0.50 * fma3(Wb.y, q.x, -Wb.x, q.y, Wb.z, q.w);
    qd.w = 0.50 * fma3(-Wb.x, q.x, -Wb.y, q.y, -Wb.z, q.z);
    qdd.x = fma2(0.50, fma3(Wdb.x, q.w, -Wdb.y, q.z, Wdb.z, q.y), 0.50, fma3(Wb.x, qd.w, -Wb.y, qd.z, Wb.z, qd.y));
    qdd.y = fma2(0.50, fma3(Wdb.x, q.z, Wdb.y, q.w, -Wdb.z, q.x), 0.50, fma3(Wb.x, qd.z, Wb.y, qd.w, -Wb.z, qd.x));
    qdd.z = fma2(0.50, fma3(Wdb.y, q.x, -Wdb.x, q.y, Wdb.z, q.w), 0.50, fma3(Wb.y, qd.x, -Wb.x, qd.y, Wb.z, qd.w));
    qdd.w = fma2(0.50, fma3(-Wdb.x, q.x, -Wdb.y, q.y, -Wdb.z, q.z), 0.50, fma3(-Wb.x, qd.x, -Wb.y, qd.y, -Wb.z, qd.z));
    const double h2 = 0.5 * Dt * Dt;
    r.x = __fma_rn(h2, qdd.x, __fma_rn(Dt, qd.x, q.x));
    r.y = __fma_rn(h2, qdd.y, __fma_rn(Dt, qd.y, q.y));
    r.z = __fma_rn(h2, qdd.z, __fma_rn(Dt, qd.z, q.z));
    r.w = __fma_rn(h2, qdd.w, __fma_rn(Dt, qd.w, q.w));
    const double inv = 1.0 / sqrt(__fma_rn(r.w, r.w, fma3(r.x, r.x, r.y, r.y, r.z, r.z)));
    r.x *= inv; r.y *= inv; r.z *= inv; r.w *= inv;
    return r;
}

// The contact slots of one subsphere, n force and torque pairs from p on: its
// near front entries, then its near back entries, in row order
// (SumContForce_clump, src/dem_force_clump.cu:165-191, sums a subsphere's
// front entries, then its back entries); the loads of a few slots are in
// flight together.
template <typename R>
__device__ __forceinline__ void slot_sum(const R4<R>* __restrict__ p, int n, V3<R>& F, V3<R>& T) {
    constexpr int U = sizeof(R) == 4 ? 4 : 2;
    F = v3<R>(0, 0, 0);
    T = F;
#pragma unroll 1
    for (int e = 0; e < n; e += U) {
        R4<R> f[U], t[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (e + u < n) ld_pair(p + 2 * (e + u), f[u], t[u]);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (e + u < n) {
                F = F + xyz<R>(f[u]);
                T = T + xyz<R>(t[u]);
            }
    }
}

// F / M + gravity and the half-kick v + h a
__device__ __forceinline__ V3<double> linear_acc(V3<double> F, double invM, double grav) {
    return v3(__dmul_rn(invM, F.x), __dmul_rn(invM, F.y), __fma_rn(invM, F.z, grav));
}
__device__ __forceinline__ V3<double> kick(V3<double> v, double h, V3<double> a) {
    return v3(__fma_rn(h, a.x, v.x), __fma_rn(h, a.y, v.y), __fma_rn(h, a.z, v.z));
}
__device__ __forceinline__ V3<double> shfl3(V3<double> v, int src) {
    return v3(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src), __shfl_sync(0xffffffffu, v.z, src));
}

// The work of one warp of the lane table (see above); every lane of the warp
// calls it with its record (ta: subsphere (-1: none), member slot, clump,
// members << 5 | first lane; tb: scene, first contact slot, slots) and the
// scene's parameters.  Returns whether the lane's subsphere has moved past its
// rebuild threshold.  SPH: the build for batches with a sphere-driver scene
// (ScenePar::sphere); the clump path's build carries none of that code.
// EARLY: the pose's records are loaded with the first ones (where registers
// allow).
template <typename R, bool SPH, bool EARLY>
__device__ __forceinline__ bool clump_warp(const Dev& d, const ScenePar& P, int4 ta, int4 tb, int do_pre, int post,
                                           int L) {
    const int lane = threadIdx.x & 31;
    const bool isc = ta.z >= 0;
    const int k = isc ? ta.z : 0, sc = tb.x;
    const int head = ta.w & 31, nm = ta.w >> 5;
    const bool stops = d.has_stops;
    const bool pre_k = isc && (stops ? scene_pre(d.dyn[sc], do_pre, L) : do_pre != 0);
    const bool post_k = isc && (stops ? scene_post(d.dyn[sc], post, L) : post != 0);
    // a warp whose clumps all belong to scenes standing still has no work
    if (stops && !__any_sync(0xffffffffu, pre_k || post_k)) return false;
    int2 im = make_int2(ta.x, ta.y), sl = make_int2(tb.y, tb.z);
    double4 cp = ld32(d.cpos + k), cv = ld32(d.cvel + k), cw = ld32(d.cw + k), cq = ld32(d.cq + k);
    const double4 pr = ld32(d.cinv + k);            // the reciprocals 1/I, 1/M
    const double Dt = P.dt, grav = P.gravity;
    double4 lo = make_double4(0, 0, 0, 0), c = lo;
    if (EARLY && im.x >= 0) {
        lo = ld32(d.lom + im.y);
        c = ld32(d.cum + im.y);
    }
    const int most = __reduce_max_sync(0xffffffffu, nm);   // members of the warp's largest clump
    double4 ps = make_double4(0, 0, 0, 0);
    V3<double> F = v3(0.0, 0.0, 0.0), T = F;
    if (post) {
        for (int c0 = 0;; c0 += 32) {
            V3<double> f = v3(0.0, 0.0, 0.0), t = f;
            const int i = im.x;
            if (i >= 0) {
                const uint16_t bb = d.bbits[i];
                ps = ld32(d.posr + i);
                V3<R> fr, tr, fw, tw;   // the boundary's share is on its way while the slots are summed
                if (bb) {
                    const R4<R>* fbd = (const R4<R>*)d.fbnd;
                    fw = xyz<R>(fbd[i]);
                    tw = xyz<R>(fbd[(size_t)d.N + i]);
                }
                slot_sum<R>((const R4<R>*)d.slots + 2 * (size_t)sl.x, sl.y, fr, tr);
                if (bb) {
                    fr = fr + fw;
                    tr = tr + tw;
                }
                const V3<double> r = v3(ps.x - cp.x, ps.y - cp.y, ps.z - cp.z);
                f = v3((double)fr.x, (double)fr.y, (double)fr.z);
                t.x = __dadd_rn((double)tr.x, fma2(r.y, f.z, -r.z, f.y));
                t.y = __dadd_rn((double)tr.y, fma2(r.z, f.x, -r.x, f.z));
                t.z = __dadd_rn((double)tr.z, fma2(r.x, f.y, -r.y, f.x));
            }
            const int mq = min(most - c0, 32);
            for (int q = 0; q < mq; q++) {
                const V3<double> fq = shfl3(f, head + q), tq = shfl3(t, head + q);
                if (c0 + q < nm) {
                    if (c0 + q == 0) { F = fq; T = tq; }
                    else { F = F + fq; T = T + tq; }
                }
            }
            if (c0 + 32 >= most) break;
            // a clump of more than 32 members: the next ones of its list
            im = make_int2(-1, 0);
            if (c0 + 32 + lane < nm) {
                im = d.mo[d.mem_start[k] + c0 + 32 + lane];
                sl = d.nsl[im.y];
            }
        }
        if (post_k) {
            if (nm > 0) {
                if (lane == head) {
                    if (!(isfinite(F.x) && isfinite(F.y) && isfinite(F.z) && isfinite(T.x) && isfinite(T.y) &&
                          isfinite(T.z)))
                        atomicOr(&d.dyn[sc].err, ERR_NONFINITE);
                    st32(d.cF + k, make_double4(F.x, F.y, F.z, 0.0));
                    st32(d.cT + k, make_double4(T.x, T.y, T.z, 0.0));
                }
            } else {
                F = xyzd(d.cF[k]);
                T = xyzd(d.cT[k]);
            }
        }
        // split driver: only Type 0 takes the closing half-kick
        // (src/dem_integrate_withglue.cu:140)
        if (post_k && !(SPH && (P.sphere & SPH_KINDS) && (d.kind[k] & 3) != 0)) {
            const V3<double> v = kick(xyzd(cv), 0.5 * Dt, linear_acc(F, pr.w, grav));
            const V3<double> o = kick(xyzd(cw), 0.5 * Dt, v3(__dmul_rn(pr.x, T.x), __dmul_rn(pr.y, T.y), __dmul_rn(pr.z, T.z)));
            cv.x = v.x; cv.y = v.y; cv.z = v.z;
            cw.x = o.x; cw.y = o.y; cw.z = o.z;
        }
    } else {
        F = xyzd(d.cF[k]);
        T = xyzd(d.cT[k]);
        if (im.x >= 0) ps = ld32(d.posr + im.x);
    }
    if (post_k && !pre_k && lane == head) {   // closing half-kick only (sync, or the scene's last step)
        st32(d.cvel + k, cv);
        st32(d.cw + k, cw);
    }
    if (!pre_k) return false;
    if (SPH && (P.sphere & SPH_KIN) && nm > 0) {
        // the sphere drivers' first half-kick and attitude leave the
        // intruder out (src/dem_integrate.cu:20-21,72); one member
        const int i = im.x;
        if ((d.bbits[i] >> SLOT_INTR) & 1) {
            const R4<R>* fi = (const R4<R>*)d.fint;
            const R4<R> a = fi[i], b = fi[(size_t)d.N + i];
            F = F - v3((double)a.x, (double)a.y, (double)a.z);
            T = T - v3((double)b.x, (double)b.y, (double)b.z);
        }
    }
    const double4 cp_old = cp;
    const V3<double> ac = linear_acc(F, pr.w, grav);
    const V3<double> al = v3(__dmul_rn(pr.x, T.x), __dmul_rn(pr.y, T.y), __dmul_rn(pr.z, T.z));
    const double h2 = 0.5 * Dt * Dt;
    // (the sphere drivers' scenes fuse the other product)
    const bool sph = SPH && P.sphere;
    cp.x = __dadd_rn(cp.x, sph ? fma2(Dt, cv.x, h2, ac.x) : fma2(h2, ac.x, Dt, cv.x));
    cp.y = __dadd_rn(cp.y, sph ? fma2(Dt, cv.y, h2, ac.y) : fma2(h2, ac.y, Dt, cv.y));
    cp.z = __dadd_rn(cp.z, fma2(Dt, cv.z, h2, ac.z));
    V3<double> v = kick(xyzd(cv), 0.5 * Dt, ac), wv = kick(xyzd(cw), 0.5 * Dt, al);
    // attitude with the half-kicked angular velocity
    double4 q = quat_step(cq, wv, al, Dt);
    if (SPH && (P.sphere & SPH_KINDS)) {
        // split driver (src/dem_integrate_withglue.cu:3-110).  Its call
        // passes the original index where the first half-kick expects
        // Type (src/dem_simulation_split.cu:84-85 against
        // src/dem_integrate_withglue.cu:113-114), so the kick and the
        // move go by the body's original index (bits 2-3: 0 free, 1
        // driven at (-0.2 y, -0.2 x, 0), 2 or more still) and the
        // attitude by its Type (bits 0-1: turns only for Type 0)
        const int kd = d.kind[k], ka = kd & 3, kb = (kd >> 2) & 3;
        if (kb != 0) {
            cp = cp_old;
            wv = xyzd(cw);
            v = xyzd(cv);
            if (kb == 1) {
                v = v3(-0.2 * cp_old.y, -0.2 * cp_old.x, 0.0);
                cp.x += Dt * v.x; cp.y += Dt * v.y; cp.z += Dt * v.z;
            }
            if (ka == 0) q = quat_step(cq, wv, al, Dt);
        }
        if (ka != 0) q = cq;
    }
    if (lane == head) {
        st32(d.cpos + k, cp);
        st32(d.cvel + k, make_double4(v.x, v.y, v.z, 0.0));
        st32(d.cw + k, make_double4(wv.x, wv.y, wv.z, 0.0));
        st32(d.cq + k, q);
    }
    // ---- the member's pose
    double thr = P.thresh;
    bool moved = false;
    for (int c0 = 0; c0 < nm; c0 += 32) {
        if (nm > 32) {   // a warp of its own: the members once more
            if (c0 + lane >= nm) break;
            im = d.mo[d.mem_start[k] + c0 + lane];
            ps = ld32(d.posr + im.x);
        }
        if (!EARLY || nm > 32) {
            lo = ld32(d.lom + im.y);
            c = ld32(d.cum + im.y);
        }
        const V3<double> arm = rot_b2w(q, v3(lo.x, lo.y, lo.z));
        const V3<double> p = v3(__dadd_rn(cp.x, arm.x), __dadd_rn(cp.y, arm.y), __dadd_rn(cp.z, arm.z));
        const V3<double> cn = v3((c.x + p.x) - ps.x, (c.y + p.y) - ps.y, (c.z + p.z) - ps.z);
        st32(d.cum + im.y, make_double4(cn.x, cn.y, cn.z, 0.0));
        st32(d.posr + im.x, make_double4(p.x, p.y, p.z, ps.w));
        st32(d.kin + im.y, make_double4(arm.x, arm.y, arm.z, lo.w));   // world arm, mass
        if (SPH && (P.sphere & SPH_KINDS))   // split driver: the free body of the first half-kick at 0.1 r
            thr = ((d.kind[k] >> 2) & 3) == 0 ? 0.10 * ps.w : INFINITY;   // (src/dem_integrate_withglue.cu:41)
        if (len_floor(cn) > thr) {
            SceneDyn& y = d.dyn[sc];
            if (!*(volatile int*)&y.rebuild) atomicExch(&y.rebuild, 1);
            if (!*(volatile int*)d.any_rebuild) atomicExch(d.any_rebuild, 1);
            moved = true;
        }
    }
    return moved;
}

// the intruder and the step count of scene s (one thread)
__device__ __forceinline__ void scene_step(const Dev& d, int s, int do_pre, int post, int L) {
    const ScenePar& P = d.par[s];
    SceneDyn& y = d.dyn[s];
    const double Dt = P.dt;
    const bool pre_s = scene_pre(y, do_pre, L), post_s = scene_post(y, post, L);
    if (post_s) {
        long long* fx = (long long*)&y.ifix[0];
        V3<double> tf = v3(fx[0] / FIX_F, fx[1] / FIX_F, fx[2] / FIX_F);
        V3<double> tt = v3(fx[3] / FIX_T, fx[4] / FIX_T, fx[5] / FIX_T);
        for (int c = 0; c < 6; c++) fx[c] = 0;
        y.totF[0] = tf.x; y.totF[1] = tf.y; y.totF[2] = tf.z;
        y.totT[0] = tt.x; y.totT[1] = tt.y; y.totT[2] = tt.z;
        if (P.has_intr) {
            if (P.intr_wait && y.intr_state == 1) y.intr_state = 2;
            V3<double> reac = v3(-tf.x, -tf.y, -tf.z);
            if (P.intr_motion == 1 && (!P.intr_wait || y.intr_state != 0)) {
                V3<double> a = (1.0 / P.intr_mass) * reac;
                a.z = a.z + P.gravity;
                for (int c = 0; c < 3; c++) y.intr_v[c] += (0.5 * Dt) * (&a.x)[c];
            }
            y.reaction[0] = reac.x; y.reaction[1] = reac.y; y.reaction[2] = reac.z;
            y.reaction_t[0] = tt.x; y.reaction_t[1] = tt.y; y.reaction_t[2] = tt.z;
            double* ring = d.ring + ((size_t)s * d.ring_len + (y.step % d.ring_len)) * 6;
            ring[0] = reac.x; ring[1] = reac.y; ring[2] = reac.z;
            ring[3] = tt.x; ring[4] = tt.y; ring[5] = tt.z;
        }
        y.step += 1;
    }
    if (do_pre) y.frozen = !pre_s;
    if (pre_s && P.has_intr) {
        if (P.intr_motion == 1 && (!P.intr_wait || y.intr_state != 0)) {
            V3<double> a = (-1.0 / P.intr_mass) * v3(y.totF[0], y.totF[1], y.totF[2]);
            a.z = a.z + P.gravity;
            for (int c = 0; c < 3; c++) {
                y.intr_p[c] = (y.intr_p[c] + Dt * y.intr_v[c]) + (0.5 * Dt * Dt) * (&a.x)[c];
                y.intr_v[c] = y.intr_v[c] + (0.5 * Dt) * (&a.x)[c];
            }
        } else {
            for (int c = 0; c < 3; c++) y.intr_p[c] = y.intr_p[c] + Dt * y.intr_v[c];
        }
    }
}

template <typename R, bool SPH>
__global__ void __launch_bounds__(CL_THREADS, NBC_CLUMP_MINB) k_clump(const Dev* __restrict__ dp, int do_pre,
                                                                      cudaGraphConditionalHandle cond, int use_cond) {
    const Dev& d = *dp;
    if (*d.halt) return;   // a rebuild ran out of pair capacity: the host finishes that step
    const int post = *d.post_pending;
    const int L = *d.lstep;   // written only by the last block, after every block has read it
    if (do_pre && blockIdx.x == 0 && threadIdx.x == 0) {
        *d.hgen += 1;
        *d.gstep += 1;
    }
    const int w = blockIdx.x * CL_WARPS + (threadIdx.x >> 5);
    if (w < d.W) {
        int4 ta, tb;
        ld_rec(d.lrec + 2 * (size_t)(w * 32 + (threadIdx.x & 31)), ta, tb);
        clump_warp<R, SPH, false>(d, d.par[tb.x], ta, tb, do_pre, post, L);
    } else {
        const int s = (w - d.W) * 32 + (threadIdx.x & 31);
        if (s < d.S) scene_step(d, s, do_pre, post, L);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(d.kc_done, 1) == (int)gridDim.x - 1) {
            *d.kc_done = 0;
            if (do_pre) *d.lstep = L + 1;
            if (use_cond) cudaGraphSetConditional(cond, atomicAdd(d.any_rebuild, 0) ? 1u : 0u);
        }
    }
}

// Clump records (old: the caller's number of each): the n clumps from `first`
// on, a scene's, out of the engine as packed doubles, ready to be copied to the
// caller's arrays: for each src with a w, n times w doubles one after the other.
struct ClumpArrays {
    const double4* src[6];
    int w[6];
    int n;
};
static __global__ void k_clumps_out(ClumpArrays a, const int* __restrict__ old, int first, int n,
                                    double* __restrict__ dst) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const int k = old[first + c] - first;
        double* o = dst;
        for (int q = 0; q < a.n; q++) {
            const double4 v = ld32(a.src[q] + first + c);
            double* p = o + (size_t)a.w[q] * k;
            p[0] = v.x; p[1] = v.y; p[2] = v.z;
            if (a.w[q] == 4) p[3] = v.w;
            o += (size_t)a.w[q] * n;
        }
    }
}
// the caller's clump, within its scene, of n subspheres
static __global__ void k_clump_ids(const int2* __restrict__ cm, const int* __restrict__ old, int first, int n,
                                   int* __restrict__ dst) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = old[cm[i].x] - first;
}
// the caller's arrays of clumps (st: position, velocity, angular velocity of 3 K
// doubles each, attitude and properties of 4 K each) into records in the engine's
// order, and the properties' reciprocals (IEEE divisions)
static __global__ void k_clumps_up(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    const double* st = (const double*)d.stage;
    const size_t K = (size_t)d.K;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d.K; c += gridDim.x * blockDim.x) {
        const size_t k = (size_t)d.cold[c];
        const double *p = st + 3 * k, *v = p + 3 * K, *w = v + 3 * K, *q = st + 9 * K + 4 * k, *m = q + 4 * K;
        st32(d.cpos + c, make_double4(p[0], p[1], p[2], 0.0));
        st32(d.cvel + c, make_double4(v[0], v[1], v[2], 0.0));
        st32(d.cw + c, make_double4(w[0], w[1], w[2], 0.0));
        st32(d.cq + c, make_double4(q[0], q[1], q[2], q[3]));
        st32(d.cprop + c, make_double4(m[0], m[1], m[2], m[3]));
        st32(d.cinv + c,
             make_double4(__ddiv_rn(1.0, m[0]), __ddiv_rn(1.0, m[1]), __ddiv_rn(1.0, m[2]), __ddiv_rn(1.0, m[3])));
    }
}
// body offset and mass (so) into the member's slot, position and radius (sp)
// into the subsphere's record: of both 3 n doubles, then n
static __global__ void k_members_up(const double* __restrict__ so, const double* __restrict__ sp,
                                    const int2* __restrict__ cm, int n, double4* __restrict__ lom,
                                    double4* __restrict__ posr) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const size_t q = 3 * (size_t)i, w = 3 * (size_t)n + i;
        st32(lom + cm[i].y, make_double4(so[q], so[q + 1], so[q + 2], so[w]));
        st32(posr + i, make_double4(sp[q], sp[q + 1], sp[q + 2], sp[w]));
    }
}
// the member lists in subsphere order, and the clump pass's lanes (idle ones,
// then those of every clump: see Dev::lrec)
static __global__ void k_members_init(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    const int stride = gridDim.x * blockDim.x, x0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int i = x0; i < d.N; i += stride) {
        const int m = d.cm[i].y;
        d.mo[m] = make_int2(i, m);
    }
    for (int l = x0; l < 32 * d.W; l += stride) {
        d.lrec[2 * l] = make_int4(-1, 0, -1, 0);
        d.lrec[2 * l + 1] = make_int4(0, 0, 0, 0);
    }
}
static __global__ void k_lanes_init(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.K; k += gridDim.x * blockDim.x) {
        const int mb = d.mem_start[k], nm = d.mem_start[k + 1] - mb, l0 = d.clane[k];
        for (int q = 0; q < min(max(nm, 1), 32); q++) {
            const int2 v = nm ? d.mo[mb + q] : make_int2(-1, 0);
            d.lrec[2 * (l0 + q)] = make_int4(v.x, v.y, k, nm << 5 | (l0 & 31));
            d.lrec[2 * (l0 + q) + 1] = make_int4(d.csid[k], 0, 0, 0);
        }
    }
}

// ===========================================================================
// broad phase
// ===========================================================================

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// A rebuild runs over the rebuilt scenes only.  k_plan lists them (ascending)
// with prefix sums of their subsphere, cell-table and clump counts; a rebuild
// kernel walks the concatenation of the rebuilt scenes with a grid-stride
// loop and finds the scene of an element by binary search in the prefix.
// Scenes that are not rebuilt keep their order, list region and histories
// untouched, so a rebuild costs in proportion to the scenes it rebuilds.
//
// plan_find: the k in [0, n) with pre[k] <= t < pre[k + 1] (empty scenes are
// passed over).
__device__ __forceinline__ int plan_find(const int* __restrict__ pre, int n, int t) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (pre[m] <= t) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// --- exclusive scan of ints -----------------------------------------------
constexpr int SC_THREADS = 256, SC_ITEMS = 8, SC_TILE = SC_THREADS * SC_ITEMS;

// Exclusive scan over a block of NT threads (every thread calls it); sh:
// NT/32 ints.
template <int NT = SC_THREADS>
__device__ __forceinline__ int block_excl_scan(int v, int* sh, int& total) {
    static_assert(NT % 32 == 0 && NT <= 1024, "whole warps, at most 32");
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < NW ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < NW) sh[lane] = w;
    }
    __syncthreads();
    const int warp_base = warp > 0 ? sh[warp - 1] : 0;
    total = sh[NW - 1];
    __syncthreads();
    return warp_base + x - v;
}

// --- exclusive scan of ints in one launch (decoupled look-back) ----------
// One to five arrays of the same length (n, or *dn) in one launch.  Blocks
// take tiles from a ticket counter until none is left: tickets [0, tiles)
// are the tiles of the first array, [tiles, 2 tiles) those of the second,
// and so on.  A tile
// publishes its aggregate, then looks back over its array's earlier tiles
// (32 at a time, one per lane of warp 0) and sums aggregates until it meets
// an inclusive prefix, and publishes its own inclusive prefix.  A block
// takes its next ticket only after finishing its tile, so a tile waits only
// on tiles held by blocks that are running: the wait always ends.  Each wait is still
// bounded (SCAN_SPIN_LIMIT polls); a block that gives up sets *fail and
// *halt, so every later kernel of the step returns at once and the host
// reports the failure instead of using the result.  The last block of the
// grid clears the tile states and the counters for the next scan.
// ctl: [0] ticket counter, [1] finished blocks.  st: one word per ticket,
// (state << 32) | value, state 1 = aggregate, 2 = inclusive prefix.
constexpr unsigned long long SCAN_AGG = 1ull << 32, SCAN_INC = 2ull << 32;
constexpr int SCAN_SPIN_LIMIT = 1 << 22;

struct ScanArrays {
    int* a[5];
    int n;
};
static __global__ void __launch_bounds__(SC_THREADS) k_scan1(ScanArrays arrs, int n, const int* dn,
                                                            unsigned long long* __restrict__ st, int* __restrict__ ctl,
                                                            int* __restrict__ halt, int* __restrict__ fail) {
    __shared__ int sh[SC_THREADS / 32];
    __shared__ int s_ticket, s_excl, s_last;
    const int nn = dn ? *dn : n;
    const int tiles = (nn + SC_TILE - 1) / SC_TILE;
    const int narr = arrs.n;
    // a fixed grid takes tiles until none is left (the grid is set when the
    // launch is captured; the tile count is known only on the device)
    for (;;) {
        if (threadIdx.x == 0) s_ticket = atomicAdd(&ctl[0], 1);
        __syncthreads();
        const int tk = s_ticket;
        __syncthreads();
        if (tk >= narr * tiles) break;
        const int arr = tk / tiles;
        const int b = tk - arr * tiles;      // tile of its array
        int* __restrict__ a = arrs.a[arr];
        unsigned long long* __restrict__ sa = st + (size_t)arr * tiles;
        const int base = b * SC_TILE + threadIdx.x * SC_ITEMS;
        // eight items a thread in one access (the arrays start on 256 bytes;
        // one by one: 12.8 us instead of 8.8 for five arrays of 200,000)
        static_assert(SC_ITEMS == 8, "a 32-byte access per thread");
        const bool whole = base + SC_ITEMS <= nn;
        int v[SC_ITEMS], sum = 0;
        if (whole) {
            int4 p, q;
            ld_rec((const int4*)(a + base), p, q);
            v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
            v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < SC_ITEMS; j++) v[j] = base + j < nn ? a[base + j] : 0;
        }
#pragma unroll
        for (int j = 0; j < SC_ITEMS; j++) sum += v[j];
        int total;
        int ex = block_excl_scan(sum, sh, total);
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int excl = 0;
            if (b == 0) {
                if (lane == 0) atomicExch(&sa[0], SCAN_INC | (unsigned)total);
            } else {
                if (lane == 0) atomicExch(&sa[b], SCAN_AGG | (unsigned)total);
                bool ok = true;
                for (int j = b - 1;; j -= 32) {
                    const int t = j - lane;
                    unsigned long long w = SCAN_INC;   // before the first tile: an inclusive zero
                    if (t >= 0) {
                        int polls = 0;
                        while (((w = *(volatile unsigned long long*)&sa[t]) >> 32) == 0) {
                            if (++polls > SCAN_SPIN_LIMIT) { ok = false; w = SCAN_INC; break; }
                            __nanosleep(64);
                        }
                    }
                    const unsigned inc = __ballot_sync(0xffffffffu, (w >> 32) == 2);
                    const int upto = inc ? __ffs(inc) - 1 : 31;   // the nearest inclusive prefix ends the sum
                    int c = lane <= upto ? (int)(unsigned)w : 0;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
                    excl += c;
                    if (inc) break;
                }
                if (!__all_sync(0xffffffffu, ok) && lane == 0) {
                    atomicExch(fail, WAIT_SCAN);
                    atomicExch(halt, 1);
                }
                if (lane == 0) atomicExch(&sa[b], SCAN_INC | (unsigned)(excl + total));
            }
            if (lane == 0) s_excl = excl;
        }
        __syncthreads();
        ex += s_excl;
#pragma unroll
        for (int j = 0; j < SC_ITEMS; j++) {
            const int x = v[j];
            v[j] = ex;
            ex += x;
        }
        if (whole) {
            st_rec((int4*)(a + base), make_int4(v[0], v[1], v[2], v[3]), make_int4(v[4], v[5], v[6], v[7]));
        } else {
#pragma unroll
            for (int j = 0; j < SC_ITEMS; j++)
                if (base + j < nn) a[base + j] = v[j];
        }
    }
    // every block has taken its ticket and is done with the tile states
    // once the finished count reaches the grid: the last one resets them
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&ctl[1], 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        for (int k = threadIdx.x; k < narr * tiles; k += SC_THREADS) st[k] = 0ull;
        if (threadIdx.x == 0) {
            ctl[0] = 0;
            ctl[1] = 0;
        }
    }
}

// warps of the clump pass's table that hold lanes of a scene
__device__ __forceinline__ int table_warps(const Dev& d, const ScenePar& P) {
    const int c0 = P.clump_off, c1 = c0 + P.nclump - 1, n1 = d.mem_start[c1 + 1] - d.mem_start[c1];
    return (d.clane[c1] + min(max(n1, 1), 32) - 1) / 32 - d.clane[c0] / 32 + 1;
}
__device__ __forceinline__ void plan_totals(const Dev& d, int ns, int nsub, int ncell, int nwarp) {
    d.psub[ns] = nsub;
    d.pcell[ns] = ncell;
    d.pwarp[ns] = nwarp;
    d.plan[PL_NS] = ns;
    d.plan[PL_T] = nsub;
    d.plan[PL_TC] = ncell;
    d.plan[PL_T1] = nsub + 1;
    d.plan[PL_TW] = nwarp;
    d.plan[PL_TC1] = ncell + 1;
}

// The plan of a rebuild (one block; a single scene's is made by k_hash).  Rebuilt scenes are listed in ascending
// order; their cell keys (cell_off + local cell) ascend with the scene, so
// sorting the concatenation of their subspheres keeps every scene in its own
// range.
static __global__ void __launch_bounds__(SC_THREADS) k_plan(const Dev* __restrict__ dp) {
    __shared__ int sh[SC_THREADS / 32];
    const Dev& d = *dp;
    if (*d.halt) return;
    int ns = 0, nsub = 0, ncell = 0, nwarp = 0;
    for (int b = 0; b < d.S; b += SC_THREADS) {
        const int s = b + threadIdx.x;
        const bool f = s < d.S && d.dyn[s].rebuild;
        int a1 = 0, a2 = 0, a3 = 0;
        if (f) {
            const ScenePar& P = d.par[s];
            a1 = P.nsub;
            a2 = P.cellnum + 1;
            a3 = table_warps(d, P);
        }
        if (s < d.S) d.need[s] = -1;
        int t0, t1, t2, t3;
        const int e0 = block_excl_scan(f ? 1 : 0, sh, t0);
        const int e1 = block_excl_scan(a1, sh, t1);
        const int e2 = block_excl_scan(a2, sh, t2);
        const int e3 = block_excl_scan(a3, sh, t3);
        if (f) {
            d.pscene[ns + e0] = s;
            d.psub[ns + e0] = nsub + e1;
            d.pcell[ns + e0] = ncell + e2;
            d.pwarp[ns + e0] = nwarp + e3;
        }
        ns += t0;
        nsub += t1;
        ncell += t2;
        nwarp += t3;
    }
    if (threadIdx.x == 0) plan_totals(d, ns, nsub, ncell, nwarp);
}

#define NBC_GRID_STRIDE(t, n) for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < (n); t += gridDim.x * blockDim.x)

// Cells on faces.  The reference sorts by floor((x - origin) / cell) and, on a
// single-level grid, centres its search on floor((x - origin) * (1 / cell))
// (src/dem_grid.cu:155-202,466-552); its hierarchical search divides.  For a
// coordinate on a cell's face, or within rounding of it, the two can differ;
// lattices at rest with round radii are full of such coordinates, a settled bed
// has none.  k_search finds cells by a product and takes the rows before a
// subsphere's own cell as sorted before it, so it needs them equal.  k_hash
// compares them: a rebuild in which some differ (or were clamped into the grid)
// sets plan[PL_FACE] and is searched by k_search_faces.  On coarser levels than
// a subsphere's own it compares them where the cells are no larger than the
// reach (ScenePar::tight); in larger ones both find every pair.
__device__ __forceinline__ int cell_coord(double x, double c) { return (int)floor(x / c); }
// whether the product with inv = 1 / c gives another cell than the quotient (it
// is off by less than 2^-50 of itself, 2^-19 at 2^31 cells)
__device__ __forceinline__ bool cells_differ(double x, double c, double inv) {
    const double t = x * inv;
    return !(fabs(t - rint(t)) > 1e-5) && (int)floor(t) != cell_coord(x, c);
}

// GetParticleCellIndex_cuk (src/dem_grid.cu:155-202); hierarchical variant
// GetParticleCellIndex_hGrid_cuk (src/dem_hgrid.cu:205-242) with the
// out-of-box bucket kept inside the scene's cell range.  Element t of the
// rebuilt concatenation: kA[t] = its cell's index u in the rebuilt scenes'
// cell table (pcell[k] + local cell), vA[t] = its arrival among the cell's
// elements; ccnt[u] counts them.
//
// The stable sort by cell (the reference sorts with CUB's stable radix
// sort, src/dem_grid.cu:278-305) is a counting sort: the scan of ccnt gives
// each cell's first sorted slot, k_cscatter drops every element into its
// cell's range, and k_order finds each element's place among the cell's
// elements by counting the smaller ones -- the order a stable sort keeps --
// and moves the element there.
//
// A single scene's plan is known to every block and written for the later
// kernels by the first one: a launch less, and with the commit in k_rows two
// (53,000 subspheres in FP64: 35.9 -> 35.3 us a step, 1,000,000: 425 -> 416).
static __global__ void k_hash(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    const bool one = d.S == 1, all = one && d.dyn[0].rebuild;
    const int T = one ? (all ? d.par[0].nsub : 0) : d.plan[PL_T], ns = one ? 1 : d.plan[PL_NS];
    if (one && blockIdx.x == 0 && threadIdx.x == 0) {
        const ScenePar& P = d.par[0];
        d.need[0] = -1;
        d.pscene[0] = d.psub[0] = d.pcell[0] = d.pwarp[0] = 0;
        if (all) plan_totals(d, 1, P.nsub, P.cellnum + 1, table_warps(d, P));
        else plan_totals(d, 0, 0, 0, 0);
    }
    NBC_GRID_STRIDE(t, T) {
        const int k = one ? 0 : plan_find(d.psub, ns, t);
        const ScenePar& P = d.par[one ? 0 : d.pscene[k]];
        const int i = P.sub_off + (one ? t : t - d.psub[k]);
        const double4 p = ld32(d.posr + i);
        const double x = p.x - P.origin[0], y = p.y - P.origin[1], z = p.z - P.origin[2];
        int local;
        bool face = false;
        if (P.levels <= 1) {
            if (p.z >= P.box_hi[2] || p.y >= P.box_hi[1] || p.x >= P.box_hi[0] ||
                p.z < P.box_lo[2] || p.y < P.box_lo[1] || p.x < P.box_lo[0]) {
                local = P.cellnum - 1;
            } else {
                const int cx = clampi(cell_coord(x, P.cell[0]), 0, P.gdim[0] - 1);
                const int cy = clampi(cell_coord(y, P.cell[1]), 0, P.gdim[1] - 1);
                const int cz = clampi(cell_coord(z, P.cell[2]), 0, P.gdim[2] - 1);
                face = cx != (int)floor(x * P.icell[0]) || cy != (int)floor(y * P.icell[1]) ||
                       cz != (int)floor(z * P.icell[2]);
                local = cz * P.gdim[1] * P.gdim[0] + cy * P.gdim[0] + cx;
                local = clampi(local, 0, P.cellnum - 1);
            }
        } else {
            if (p.z > P.box_hi[2] || p.y > P.box_hi[1] || p.x > P.box_hi[0] ||
                p.z < P.box_lo[2] || p.y < P.box_lo[1] || p.x < P.box_lo[0]) {
                local = P.cellnum - 1;
            } else {
                const int lv = d.level[i];
                const double c = P.lcell[lv], in = P.licell[lv];
                const int cx = clampi(cell_coord(x, c), 0, P.ldim[lv][0] - 1);
                const int cy = clampi(cell_coord(y, c), 0, P.ldim[lv][1] - 1);
                const int cz = clampi(cell_coord(z, c), 0, P.ldim[lv][2] - 1);
                face = cx != (int)floor(x * in) || cy != (int)floor(y * in) || cz != (int)floor(z * in);
                if (P.tight)   // the coarser levels it searches
                    for (int l = 0; l < lv; l++)
                        face |= cells_differ(x, P.lcell[l], P.licell[l]) | cells_differ(y, P.lcell[l], P.licell[l]) |
                                cells_differ(z, P.lcell[l], P.licell[l]);
                local = P.loff[lv] + (cz * P.ldim[lv][1] * P.ldim[lv][0] + cy * P.ldim[lv][0] + cx);
            }
        }
        if (face) d.plan[PL_FACE] = 1;
        const int u = (one ? 0 : d.pcell[k]) + local;
        d.kA[t] = u;
        d.vA[t] = atomicAdd(&d.ccnt[u], 1);
    }
}

// every element into its cell's range (in order of arrival within the cell);
// the list's counters start at zero
static __global__ void k_cscatter(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    const int T = d.plan[PL_T];
    NBC_GRID_STRIDE(t, T + 1) {
        d.cnt_f[t] = 0;
        d.cnt_b[t] = 0;
        d.cnt_nf[t] = 0;
        d.cnt_ns[t] = 0;
        d.xcnt[t] = 0;
        if (t == T) break;
        d.fcur[t] = 0;
        d.vB[d.ccnt[d.kA[t]] + d.vA[t]] = t;
    }
}

// Boundary candidates.  Walls do not move (their velocity enters only the
// contact law), and between two rebuilds of a scene every subsphere stays
// within Thresh of where it was at the rebuild, so a subsphere farther than
// 2 Thresh from every wall region at a rebuild cannot touch a wall before
// the next one.  Each rebuild flags, per rebuilt subsphere (new order),
// whether it is within that margin of a wall -- every subsphere of a scene
// with an intruder is a candidate, the intruder moves -- and clears the wall
// contact bits of the others (they are not in contact now); k_fill lists the
// candidates in the scene's range of bidx, and k_boundary visits only them.
__device__ __forceinline__ bool bound_candidate(const ScenePar& P, double4 pp) {
    bool cand = P.has_intr;
    if (!cand && P.wall != WALL_NONE) {
        const double m = 2.0 * P.thresh * (1.0 + 1e-6) + 1e-12;
        const double r = pp.w + m;
        const double ex = pp.x - P.w_c[0], ey = pp.y - P.w_c[1], ez = pp.z - P.w_c[2];
        if (P.wall == WALL_CUBE) {
            cand = fabs(ex) + r >= P.w_half[0] * (1 - 1e-9) || fabs(ey) + r >= P.w_half[1] * (1 - 1e-9) ||
                   fabs(ez) + r >= P.w_half[2] * (1 - 1e-9);
        } else {
            const double ax = ex * P.cyl_axis[0] + ey * P.cyl_axis[1] + ez * P.cyl_axis[2];
            const double rr = ex * ex + ey * ey + ez * ez - ax * ax;
            const double in = P.cyl_R - r;
            cand = fabs(ax) + r >= P.cyl_H * (1 - 1e-9) || in <= 0 || rr >= in * in * (1 - 1e-9);
        }
    }
    return cand;
}

// Sorted slot, permutation and reorder in one pass over the scattered
// elements (SortArray_*_cuk, src/dem_grid.cu:336-437, for every persistent
// per-subsphere array at once, into the alternate buffers that k_commit makes
// current), the cell table, the boundary candidates, and the search's FP32
// copy of the positions.  A cell holds a few elements, so counting the smaller
// ones costs a few cached reads; an out-of-box bucket of n costs n^2 / 2
// reads spread over n threads.
template <typename R>
__global__ void k_order(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    const int T = d.plan[PL_T], TC = d.plan[PL_TC], ns = d.plan[PL_NS];
    const size_t N = (size_t)d.N;
    const int* __restrict__ vB = d.vB;
    NBC_GRID_STRIDE(x, T) {
        const int t = vB[x], u = d.kA[t];
        const int a = d.ccnt[u], b = d.ccnt[u + 1];
        const int k = plan_find(d.psub, ns, t);
        const ScenePar& P = d.par[d.pscene[k]];
        const int base = P.sub_off - d.psub[k];
        const int o = base + t;
        const double4 p = ld32(d.posr + o);
        int rank = 0;
        for (int y = a; y < b; y++) rank += vB[y] < t;
        const int i = base + a + rank;
        d.perm[i] = o;
        d.inv[o] = i;
        d.key2[i] = P.cell_off + (u - d.pcell[k]);
        st32(d.posr2 + i, p);
        // FP32 position from the scene's origin; w: the cutoff's share of this
        // subsphere, widened by more than the rounding of its coordinates
        // (2^-24 of each, four times over) and of the test itself
        const float fx = (float)(p.x - P.origin[0]), fy = (float)(p.y - P.origin[1]), fz = (float)(p.z - P.origin[2]);
        d.posf[i] = make_float4(fx, fy, fz,
                                1.5f * (float)p.w * (1.0f + 0x1p-19f) + 0x1p-22f * (fabsf(fx) + fabsf(fy) + fabsf(fz)));
        d.cm2[i] = d.cm[o];
        d.part_fix2[i] = d.part_fix[o];
        d.level2[i] = d.level[o];
        const bool cand = bound_candidate(P, p);
        d.xcnt[i - base] = cand;
        const uint16_t bits = cand ? d.bbits[o] : 0;
        d.bbits2[i] = bits;
        if (bits) {
            const R4<R>* b1 = (const R4<R>*)d.bhist;
            R4<R>* b2 = (R4<R>*)d.bhist2;
            for (int sl = 0; sl < NB_SLOTS; sl++) {
                if (!(bits & (1u << sl))) continue;  // only live histories are ever read
                for (int c = 0; c < 3; c++) b2[((size_t)sl * N + i) * 3 + c] = b1[((size_t)sl * N + o) * 3 + c];
            }
        }
    }
    // the cell table (the entry after a scene's last cell is the end of its range)
    NBC_GRID_STRIDE(u, TC) {
        const int k = plan_find(d.pcell, ns, u);
        const ScenePar& P = d.par[d.pscene[k]];
        d.cstart[P.cell_off + (u - d.pcell[k])] = P.sub_off - d.psub[k] + d.ccnt[u];
    }
}

// --- neighbour search ----------------------------------------------------
// The candidate test and the order of CreateAnei_cuk (src/dem_grid.cu:466-552):
// cells in z, y, x order over -1..1, partners ascending within a cell,
// candidate if |xi - xj|^2 < (1.5 (ri + rj))^2 in FP64; j > i goes to the
// front (owner) row of i, j < i to its back row.
//
// Hierarchical grid (CreateAnei_hGrid_cuk, src/dem_hgrid_contlist.cu:57-161):
// a subsphere searches its own level and every coarser one (level 0 is the
// coarsest); a pair across levels is owned by the coarser subsphere: the
// finer one records a back entry, the coarser one a front entry, placed after
// its same-level front entries in ascending order of the finer partner.
//
// The sorted order is level-major (coarsest first) and z, y, x within a level,
// so in both grids the owner of a pair is the subsphere with the smaller
// index, a front row is its partners in ascending order, and a back row is
// the partners j < i on i's own level in ascending order, then those of each
// coarser level, nearest level first, ascending.  Hence one half of the search
// is enough: a subsphere looks only for partners j < i (the stencil's cells up
// to its own slot, and all 27 of each coarser level), in the order of its back
// row, and counts itself into the partner's front row; k_fill hands every back
// entry to the partner's row and k_rows puts the rows in order.
//
// The three x-neighbour cells of one (z, y) stencil row hold one contiguous
// range of the sorted order.  G lanes share a subsphere: they resolve its rows
// (passing over rows and end cells that the largest cutoff on their level,
// 1.5 (ri + largest radius), cannot reach, but never at the grid's border, whose
// cells also hold what lies beyond them), walk the rows' concatenation G
// candidates at a time, and keep what passes an FP32 test (a 16-byte copy of
// the position, a cutoff widened by the rounding) in a list in shared memory;
// the list is tested in FP64, G entries at a time, and appended to the back row
// through ballots.  So the candidate loop is some thirty instructions with
// every lane busy, and the FP64 test, the flags and the counters run on full
// groups for the one candidate in eight that needs them.  50,000 clumps on five
// levels, 1.7 M pairs: 115 us (both directions with FP64 tests on 8 lanes took
// 241, and compaction, cross-level sort, reverse map, history carry and near
// rows another 250 in eight launches where k_fill and k_rows take 52 + 50).
// Half of it is the rows, a third the FP32 tests; votes with a mask per group
// instead of the whole warp's: 167 us, every lane finding its rows' levels for
// itself: 125 us, 80 or 94 registers a thread: 9 and 18% more than with 64.
//
// A subsphere in a single-level scene's last cell, where out-of-box ones are
// put, does not search; those whose stencil holds that cell list its members
// in their front rows only (no back entry), as the reference does.
constexpr int SEARCH_THREADS = 128;
constexpr int SEARCH_G = 8;                   // lanes per subsphere
constexpr int SEARCH_GROUPS = SEARCH_THREADS / SEARCH_G;
constexpr int SCR_CAP = 64;                   // scratch entries per back row
constexpr int ROW_LONG = 1, ROW_FACES = 2;     // Dev::rlong: the row is not in the scratch; made by fill_faces
constexpr int LIST_CAP = 32;                  // FP32 hits held before they are tested in FP64
constexpr int MAX_ROWS = 5 + 9 * (MAX_LEVELS - 1);
constexpr int NEAR = 0x40000000;              // scratch: the pair can touch before the next rebuild
constexpr int SUB_MASK = 0x3fffffff;

// per row that has candidates: the end of its range in the rows' concatenation,
// and the sorted index of a candidate less its place in the concatenation
struct SearchRows {
    int2 row[SEARCH_GROUPS][MAX_ROWS];
    // where the subsphere sits on each level it searches, one lane a level:
    // squared distance to the neighbour cells' faces (0 where a cell is never
    // passed over, INF where there is none), the squared reach; the centre cell,
    // the strides of the grid, the range of x neighbours
    float4 dist[SEARCH_GROUPS][MAX_LEVELS][2];   // z-, z0, z+, reach; y-, y0, y+, x-
    float xp[SEARCH_GROUPS][MAX_LEVELS];
    int4 cell[SEARCH_GROUPS][MAX_LEVELS];        // centre, stride y, stride z, (x range)
};

// FP64 test of a candidate that passed the FP32 one: 0 no pair, 1 a pair, 2 a
// near pair (see k_rows)
__device__ __forceinline__ int pair_test(double4 a, double4 b, double margin) {
    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const double d2 = fma3(dx, dx, dy, dy, dz, dz);
    const double r = a.w + b.w, lim = 1.50 * r, nlim = r + margin;
    return d2 < lim * lim ? (d2 < nlim * nlim ? 2 : 1) : 0;
}
// Near pairs: between two rebuilds of a scene every subsphere stays within
// Thresh of where it was at the rebuild (a larger displacement triggers the
// next one), so a pair whose distance at a rebuild is at least ri + rj +
// 2 Thresh cannot touch before the next one.
__device__ __forceinline__ double near_margin(const ScenePar& P) { return 2.0 * P.thresh * (1.0 + 1e-6) + 1e-12; }

// FACES (k_search_faces, and fill_faces' rows): own cells as
// the sort has them, and the reference's stencils.  A pair belongs to the list
// when the owner's stencil holds the partner's cell, and has a back entry when
// the partner's holds the owner's; across levels the finer one's stencil decides
// both.  The two disagree only on pairs about a cell apart on a single level,
// where an owner whose product lies in the next cell may list partners two cells
// on, and on subspheres outside the grid.  Where the partner alone would list
// the other there is no pair to refer to, and no entry.
//
// The rows on a single level then: two cells to each side, as far as the reach
// goes (r of 13, the last one the subsphere's own).
constexpr int FACE_ROWS = 13;
__device__ __forceinline__ bool face_row(const ScenePar& P, double4 pi, int r, int& ca, int& cb) {
    const double x = pi.x - P.origin[0], y = pi.y - P.origin[1], z = pi.z - P.origin[2], c = P.cell[0];   // cells are cubes
    const int gx = P.gdim[0], gy = P.gdim[1], gz = P.gdim[2];
    const int cx = clampi(cell_coord(x, c), 0, gx - 1), cy = clampi(cell_coord(y, c), 0, gy - 1);
    const int cz = clampi(cell_coord(z, c), 0, gz - 1);
    const int sz = r / 5 - 2, sy = r % 5 - 2;
    if (cz + sz < 0 || cy + sy < 0 || cy + sy >= gy) return false;
    const float cf = (float)c, cut = 1.5f * ((float)pi.w + P.lrmax[0]) * 1.0001f + 1e-4f * cf;
    // squared distance to the cells s away along an axis, f from the own cell's lower face
    auto dist2 = [&](int q, int n, int s, float f) {
        const float h = s < 0 ? f - (float)(s + 1) * cf : (float)s * cf - f;
        return s == 0 || q + s == 0 || q + s == n - 1 ? 0.0f : h * h;
    };
    const float rem = cut * cut - dist2(cz, gz, sz, (float)(z - cz * c)) - dist2(cy, gy, sy, (float)(y - cy * c));
    if (!(rem >= 0)) return false;
    const float fx = (float)(x - cx * c);
    int lo = max(-2, -cx), hi = min(2, gx - 1 - cx);
    while (lo < 0 && dist2(cx, gx, lo, fx) > rem) lo++;
    while (hi > 0 && dist2(cx, gx, hi, fx) > rem) hi--;
    const int m = P.cell_off + ((cz + sz) * gy + cy + sy) * gx + cx;
    ca = m + lo;
    cb = m + hi + 1;
    return true;
}
// Whose stencil holds the other's cell, of a pair j < i: 1 the owner's, 2 that
// of i.  Both when they are less than a cell apart on every axis (the cells'
// rounding is 2^-50 of a coordinate) in a box inside the grid.
__device__ __forceinline__ int face_sides(const Dev& d, const ScenePar& P, int j, double4 pj, int i, double4 pi) {
    const bool hg = P.levels > 1;
    const int l = hg ? d.level2[i] : 0;
    if (hg && d.level2[j] != l) return 3;
    const double c = hg ? P.lcell[l] : P.cell[0];
    if (P.inside && fmax(fmax(fabs(pi.x - pj.x), fabs(pi.y - pj.y)), fabs(pi.z - pj.z)) < c * (1.0 - 1e-6)) return 3;
    int sides = 3;
#pragma unroll 1
    for (int a = 0; a < 3; a++) {
        const double xj = (a == 0 ? pj.x : (a == 1 ? pj.y : pj.z)) - P.origin[a];
        const double xi = (a == 0 ? pi.x : (a == 1 ? pi.y : pi.z)) - P.origin[a];
        const int top = (hg ? P.ldim[l][a] : P.gdim[a]) - 1, uj = cell_coord(xj, c), ui = cell_coord(xi, c);
        const int mj = hg ? uj : (int)floor(xj * P.icell[a]), mi = hg ? ui : (int)floor(xi * P.icell[a]);
        if ((unsigned)clampi(ui, 0, top) - (unsigned)mj + 1u > 2u) sides &= ~1;
        if ((unsigned)clampi(uj, 0, top) - (unsigned)mi + 1u > 2u) sides &= ~2;
    }
    return sides;
}

// The stencil rows of subsphere i by the G lanes of its group (g of them):
// candidates j < i as ranges in back-row order; the number of candidates.
// Every lane of the warp calls it; `on`: the group has a subsphere.  (The
// warp's groups run in step, votes and shuffles over the whole warp: with a
// mask per group the compiler takes the groups through them one by one.)
template <bool FACES>
__device__ __forceinline__ int group_rows(const Dev& d, const ScenePar& P, bool on, int i, double4 pi, int g,
                                          SearchRows& sh, int grp) {
    constexpr int G = SEARCH_G, MAXC = (MAX_ROWS + G - 1) / G;
    const int* __restrict__ cstart = d.cstart;
    const bool hg = P.levels > 1;
    const int my = hg && on ? d.level2[i] : 0;
    const bool wide = FACES && !hg;
    const int nrows = on ? (wide ? FACE_ROWS : 5 + 9 * my) : 0, r0 = nrows * g / G, r1 = nrows * (g + 1) / G;
    int2* rows = sh.row[grp];
    __syncwarp();   // the previous rows and levels are no longer read
    if (on && g <= my) {
        const int l = my - g;
        double c0, c1, c2, i0, i1, i2;
        int gx, gy, gz, base;
        if (hg) {
            gx = P.ldim[l][0]; gy = P.ldim[l][1]; gz = P.ldim[l][2];
            base = P.cell_off + P.loff[l];
            c0 = c1 = c2 = P.lcell[l];
            i0 = i1 = i2 = P.licell[l];
        } else {
            gx = P.gdim[0]; gy = P.gdim[1]; gz = P.gdim[2];
            base = P.cell_off;
            c0 = P.cell[0]; c1 = P.cell[1]; c2 = P.cell[2];
            i0 = P.icell[0]; i1 = P.icell[1]; i2 = P.icell[2];
        }
        const double x0 = pi.x - P.origin[0], y0 = pi.y - P.origin[1], z0 = pi.z - P.origin[2];
        int cx = FACES ? cell_coord(x0, c0) : (int)floor(x0 * i0);
        int cy = FACES ? cell_coord(y0, c1) : (int)floor(y0 * i1);
        int cz = FACES ? cell_coord(z0, c2) : (int)floor(z0 * i2);
        if (FACES && g == 0) {   // on its own level
            cx = clampi(cx, 0, gx - 1);
            cy = clampi(cy, 0, gy - 1);
            cz = clampi(cz, 0, gz - 1);
        }
        const float fx = (float)(x0 - cx * c0), fy = (float)(y0 - cy * c1), fz = (float)(z0 - cz * c2);
        const float ux = (float)c0 - fx, uy = (float)c1 - fy, uz = (float)c2 - fz;
        const float cut = 1.5f * ((float)pi.w + P.lrmax[l]) * 1.0001f + 1e-4f * (float)c0;
        // a neighbour at c of g cells, h away
        auto far2 = [](int c, int g, float h) {
            return c < 0 || c >= g ? INFINITY : (c == 0 || c == g - 1 ? 0.0f : h * h);
        };
        const int xa = max(cx - 1, 0), xb = min(cx + 1, gx - 1);
        sh.dist[grp][g][0] = make_float4(far2(cz - 1, gz, fz), cz < 0 || cz >= gz ? INFINITY : 0.0f,
                                         far2(cz + 1, gz, uz), cut * cut);
        sh.dist[grp][g][1] = make_float4(far2(cy - 1, gy, fy), cy < 0 || cy >= gy ? INFINITY : 0.0f,
                                         far2(cy + 1, gy, uy),
                                         xa > 0 && xa < cx && xa < gx - 1 ? fx * fx : -1.0f);
        sh.xp[grp][g] = xb < gx - 1 && xb > cx && xb > 0 ? ux * ux : -1.0f;
        sh.cell[grp][g] = make_int4(base + (cz * gy + cy) * gx + cx, gx, gx * gy,
                                    xa > xb ? 0 : (1 << 16 | (xa - cx + 64) << 8 | (xb - cx + 64)));
    }
    __syncwarp();
    // the cells of the lane's rows first, then all their cstart loads at once
    int ca[MAXC], cb[MAXC];
#pragma unroll
    for (int k = 0; k < MAXC; k++) {
        const int r = r0 + k;
        ca[k] = -1;
        cb[k] = -1;
        if (r >= r1) continue;
        if (wide) {
            face_row(P, pi, r, ca[k], cb[k]);
            continue;
        }
        const int q = r < 5 ? 0 : 1 + (r - 5) / 9, rr = r < 5 ? r : (r - 5) % 9;
        const int sz = rr / 3 - 1, sy = rr % 3 - 1;
        const float4 fz = sh.dist[grp][q][0], fy = sh.dist[grp][q][1];
        const int4 c = sh.cell[grp][q];
        const float rem = fz.w - (sz < 0 ? fz.x : (sz ? fz.z : fz.y)) - (sy < 0 ? fy.x : (sy ? fy.z : fy.y));
        int lo = ((c.w >> 8) & 255) - 64, hi = (c.w & 255) - 64;
        if (fy.w > rem) lo = 0;
        if (sh.xp[grp][q] > rem) hi = 0;
        if (!(rem >= 0) || c.w == 0 || lo > hi) continue;
        const int m = c.x + sz * c.z + sy * c.y;
        ca[k] = m + lo;
        cb[k] = m + hi + 1;
    }
#pragma unroll
    for (int k = 0; k < MAXC; k++) {
        if (ca[k] < 0) continue;
        ca[k] = cstart[ca[k]];
        cb[k] = r0 + k == (wide ? FACE_ROWS - 1 : 4) ? i : cstart[cb[k]];
    }
    // rows with candidates, packed: (rows << 26 | candidates) summed over the lanes
    // (2^26 subspheres are 100 GB of state, without their pairs)
    constexpr int CBITS = 26;
    constexpr unsigned CMASK = (1u << CBITS) - 1u;
    static_assert(MAX_ROWS < 1 << (32 - CBITS) && FACE_ROWS <= MAX_ROWS, "the rows' count above the candidates");
    unsigned acc = 0;
#pragma unroll
    for (int k = 0; k < MAXC; k++)
        if (ca[k] >= 0 && cb[k] > ca[k]) acc += (1u << CBITS) + (unsigned)(cb[k] - ca[k]);
    unsigned inc = acc;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, inc, o, G);
        if (g >= o) inc += v;
    }
    const unsigned all = __shfl_sync(0xffffffffu, inc, G - 1, G);
    unsigned at = inc - acc;
#pragma unroll
    for (int k = 0; k < MAXC; k++)
        if (ca[k] >= 0 && cb[k] > ca[k]) {
            const int c = (int)(at & CMASK);
            rows[at >> CBITS] = make_int2(c + cb[k] - ca[k], ca[k] - c);
            at += (1u << CBITS) + (unsigned)(cb[k] - ca[k]);
        }
    __syncwarp();
    return (int)(all & CMASK);
}

// the members of a single-level scene's last cell when subsphere i's stencil
// holds it (its front-only partners are among them): their range
__device__ __forceinline__ int2 last_cell(const Dev& d, const ScenePar& P, double4 pi) {
    if (P.levels > 1 || (int)floor((pi.x - P.origin[0]) * P.icell[0]) + 1 < P.gdim[0] - 1 ||
        (int)floor((pi.y - P.origin[1]) * P.icell[1]) + 1 < P.gdim[1] - 1 ||
        (int)floor((pi.z - P.origin[2]) * P.icell[2]) + 1 < P.gdim[2] - 1)
        return make_int2(0, 0);
    const int b = P.cell_off + P.cellnum - 1;
    return make_int2(d.cstart[b], d.cstart[b + 1]);
}

// the subsphere of element t of the rebuilt concatenation and its scene
struct PlanItem {
    int k, s, i;
};
__device__ __forceinline__ PlanItem plan_item(const Dev& d, int ns, int t) {
    PlanItem r;
    r.k = plan_find(d.psub, ns, t);
    r.s = d.pscene[r.k];
    r.i = d.par[r.s].sub_off + (t - d.psub[r.k]);
    return r;
}
__device__ __forceinline__ bool searches(const Dev& d, const ScenePar& P, int i) {
    return d.key2[i] != P.cell_off + P.cellnum - 1;   // out-of-box subspheres do not search
}

// The search: back rows into the scratch (rlong set where they do not fit or
// there are front-only partners), their lengths (cnt_b), those of
// the front rows (cnt_f) and of the near front rows (cnt_nf), and the contact
// slots of each member slot (cnt_ns: near entries of both rows).
template <bool FACES>
__device__ __forceinline__ void search_rows(const Dev& d, SearchRows& sh, int (*s_buf)[LIST_CAP]) {
    constexpr int G = SEARCH_G;
    const int T = d.plan[PL_T], ns = d.plan[PL_NS];
    const int g = threadIdx.x % G, grp = threadIdx.x / G;
    const int gshift = (threadIdx.x & 31) & ~(G - 1);
    constexpr unsigned GM = (1u << G) - 1u;
    const unsigned lt = (1u << g) - 1u;
    const double4* __restrict__ posr = d.posr2;
    const float4* __restrict__ posf = d.posf;
    const int2* __restrict__ cm = d.cm2;
    int* __restrict__ cnt_f = d.cnt_f;
    int* __restrict__ cnt_nf = d.cnt_nf;
    int* __restrict__ cnt_ns = d.cnt_ns;
    int2* rows = sh.row[grp];
    int* buf = s_buf[grp];
    constexpr unsigned FULL = 0xffffffffu;
    for (int b0 = blockIdx.x * SEARCH_GROUPS + (grp & ~3); b0 < T; b0 += gridDim.x * SEARCH_GROUPS) {
        const int t = b0 + (grp & 3);
        const PlanItem it = plan_item(d, ns, min(t, T - 1));
        const int i = it.i, tb = min(t, T - 1) - i;
        const ScenePar& P = d.par[it.s];
        const bool on = t < T && searches(d, P, i);
        const double4 pi = ld32(posr + i);
        const float4 pf = posf[i];
        const int2 ci = cm[i];
        const int total = group_rows<FACES>(d, P, on, i, pi, g, sh, grp);
        const int most = __reduce_max_sync(FULL, total);
        // the candidates in order, G at a time (the next ones' positions in
        // flight): what passes goes to the list through a vote, and a list that
        // cannot take another G is tested in FP64 and emptied
        const double margin = near_margin(P);
        int* __restrict__ scr = d.scr + (size_t)i * SCR_CAP;
        int nb = 0, near = 0, n = 0, r = 0, jn = -1;
        bool alone = false;   // (FACES) some entry without a back entry: the row is made by k_fill
        float4 qn = make_float4(0, 0, 0, 0);
        auto next = [&](int f) {
            jn = -1;
            if (f < total) {
                int2 x = rows[r];
                while (x.x <= f) x = rows[++r];
                jn = f + x.y;
                qn = posf[jn];
            }
        };
        next(g);
        for (int f0 = 0; f0 < most; f0 += G) {
            const int j = jn;
            const float dx = pf.x - qn.x, dy = pf.y - qn.y, dz = pf.z - qn.z, w = pf.w + qn.w;
            next(f0 + G + g);
            const bool pass = j >= 0 && !(dx * dx + dy * dy + dz * dz > w * w);
            const unsigned pm = (__ballot_sync(FULL, pass) >> gshift) & GM;
            if (pass) buf[n + __popc(pm & lt)] = j;
            n += __popc(pm);
            if (f0 + G < most && !__any_sync(FULL, n > LIST_CAP - G)) continue;
            __syncwarp();
            const int list = __reduce_max_sync(FULL, n);
            for (int k0 = 0; k0 < list; k0 += G) {
                int hit = 0, k = 0;
                int2 ck = make_int2(0, 0);
                if (k0 + g < n) {
                    k = buf[k0 + g];
                    ck = cm[k];
                    hit = pair_test(ld32(posr + k), pi, margin);
                }
                int sides = 3;
                if (FACES && hit) {
                    sides = face_sides(d, P, k, ld32(posr + k), i, pi);
                    if (!(sides & 1)) hit = 0;
                    if (sides == 1) alone = true;
                }
                const bool nr = hit == 2 && ck.x != ci.x;
                const unsigned hm = (__ballot_sync(FULL, hit != 0 && sides == 3) >> gshift) & GM;
                const unsigned nm = (__ballot_sync(FULL, nr && sides == 3) >> gshift) & GM;
                if (hit) {
                    const int q = nb + __popc(hm & lt);
                    if (q < SCR_CAP && sides == 3) scr[q] = k | (ck.x == ci.x ? INTRA : 0) | (nr ? NEAR : 0);
                    atomicAdd(&cnt_f[k + tb], 1);
                    if (nr) {
                        atomicAdd(&cnt_nf[k + tb], 1);
                        atomicAdd(&cnt_ns[ck.y + tb], 1);
                    }
                }
                nb += __popc(hm);
                near += __popc(nm);
            }
            n = 0;
            __syncwarp();
        }
        bool isl = nb > SCR_CAP || alone;
        if (on) {
            const int2 lcell = last_cell(d, P, pi);
            int nx = 0, nxn = 0;
            for (int j = lcell.x + g; j < lcell.y; j += G) {
                const int hit = pair_test(pi, ld32(posr + j), margin);
                nx += hit != 0;
                nxn += hit == 2 && cm[j].x != ci.x;
            }
            if (nx) {
                isl = true;
                atomicAdd(&cnt_f[t], nx);
                if (nxn) {
                    atomicAdd(&cnt_nf[t], nxn);
                    atomicAdd(&cnt_ns[ci.y + tb], nxn);
                }
            }
            if (g == 0 && near) atomicAdd(&cnt_ns[ci.y + tb], near);
        }
        const unsigned il = (__ballot_sync(FULL, isl) >> gshift) & GM;
        if (g == 0 && t < T) {
            d.cnt_b[t] = nb;
            d.rlong[t] = il ? (FACES ? ROW_FACES : ROW_LONG) : 0;
        }
    }
}
static __global__ void __launch_bounds__(SEARCH_THREADS, 8) k_search(const Dev* __restrict__ dp) {
    __shared__ SearchRows sh;
    __shared__ int s_buf[SEARCH_GROUPS][LIST_CAP];
    const Dev& d = *dp;
    if (*d.halt) return;
    const int TC1 = d.plan[PL_TC1];
    NBC_GRID_STRIDE(u, TC1) d.ccnt[u] = 0;   // the sort's cell counts back to zero for the next rebuild
    if (!d.plan[PL_FACE]) search_rows<false>(d, sh, s_buf);
}
// The same for a rebuild with cells on faces (see cell_coord); in any other it
// returns at once, 3 us by itself and under 1% of a step in the graph.  A launch of
// its own: in k_search the second build costs the first 10% (registers), and
// dividing there for every subsphere 2 to 3%.  A lattice of 195,112 spheres at
// rest: 168 us, on three levels 118.
static __global__ void __launch_bounds__(SEARCH_THREADS) k_search_faces(const Dev* __restrict__ dp) {
    __shared__ SearchRows sh;
    __shared__ int s_buf[SEARCH_GROUPS][LIST_CAP];
    const Dev& d = *dp;
    if (*d.halt || !d.plan[PL_FACE]) return;
    search_rows<true>(d, sh, s_buf);
}

// the pairs of rebuilt scene k's new list (after the scans; a pair has one
// owner entry and, but for the front-only ones, one partner entry)
__device__ __forceinline__ int list_need(const Dev& d, int k) {
    const int a = d.psub[k], b = d.psub[k + 1];
    return max(d.cnt_f[b] - d.cnt_f[a], d.cnt_b[b] - d.cnt_b[a]);
}
// the lengths of the new lists, for the host (first list, growth)
static __global__ void k_need(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    for (int k = threadIdx.x; k < d.plan[PL_NS]; k += blockDim.x) d.need[d.pscene[k]] = list_need(d, k);
}

// The rows of k_search_faces that are not in the scratch (long ones, and those
// with an entry without a back entry), a thread each: their candidates once more.
static __device__ __forceinline__ void fill_faces(const Dev& d) {
    const int T = d.plan[PL_T], ns = d.plan[PL_NS];
    NBC_GRID_STRIDE(t, T) {
        if (d.rlong[t] != ROW_FACES) continue;
        const PlanItem it = plan_item(d, ns, t);
        const int i = it.i, tb = t - i, t0 = d.psub[it.k];
        const ScenePar& P = d.par[it.s];
        const double4 pi = ld32(d.posr2 + i);
        const int2 ci = d.cm2[i];
        const bool hg = P.levels > 1;
        const int my = hg ? d.level2[i] : 0, w = hg ? 1 : 2;
        const int base = d.dyn[it.s].pair_off, poff = base - d.cnt_f[t0];
        int kr = base + d.cnt_b[t] - d.cnt_b[t0];
        const int ke = base + d.cnt_b[t + 1] - d.cnt_b[t0];
        int kb = 2 * base + d.cnt_ns[ci.y + tb] - d.cnt_ns[t0] + d.cnt_nf[t + 1] - d.cnt_nf[t];
        const double margin = near_margin(P);
        // b into the front row of a (no row takes more than was counted)
        auto put = [&](int at, int a, int b, int h, int back) {
            const bool intra = d.cm2[a].x == d.cm2[b].x;
            const int v = intra ? INTRA : (h == 2 ? NEAR : 0);
            const int q = d.cnt_f[at] + atomicAdd(&d.fcur[at], 1);
            if (q < d.cnt_f[at + 1]) d.tmp[q + poff] = make_int2(b | v, back);
            return v;
        };
#pragma unroll 1
        for (int l = my; l >= 0; l--) {
            const bool own = l == my;
            const double c = hg ? P.lcell[l] : P.cell[0];
            const int gx = hg ? P.ldim[l][0] : P.gdim[0], gy = hg ? P.ldim[l][1] : P.gdim[1];
            const int gz = hg ? P.ldim[l][2] : P.gdim[2], c0 = P.cell_off + (hg ? P.loff[l] : 0);
            int cx = cell_coord(pi.x - P.origin[0], c), cy = cell_coord(pi.y - P.origin[1], c);
            int cz = cell_coord(pi.z - P.origin[2], c);
            if (own) {
                cx = clampi(cx, 0, gx - 1);
                cy = clampi(cy, 0, gy - 1);
                cz = clampi(cz, 0, gz - 1);
            }
            const int xa = max(cx - w, 0), xb = min(cx + w, gx - 1);
#pragma unroll 1
            for (int r = 0; r < (2 * w + 1) * (2 * w + 1) && xa <= xb; r++) {
                const int sz = r / (2 * w + 1) - w, sy = r % (2 * w + 1) - w, z = cz + sz, y = cy + sy;
                if (own && (sz > 0 || (sz == 0 && sy > 0))) break;   // sorted behind i
                if (z < 0 || z >= gz || y < 0 || y >= gy) continue;
                const int m = c0 + (z * gy + y) * gx, e = min(d.cstart[m + xb + 1], i);
#pragma unroll 1
                for (int j = d.cstart[m + xa]; j < e; j++) {
                    const double4 pj = ld32(d.posr2 + j);
                    const int h = pair_test(pj, pi, margin), sides = h ? face_sides(d, P, j, pj, i, pi) : 0;
                    if (!(sides & 1)) continue;
                    const bool back = sides == 3 && kr < ke;
                    const int v = put(j + tb, j, i, h, back ? kr : -1);
                    if (!back) continue;
                    d.L[1].bnbr[kr] = j | (v & ~NEAR);
                    if (v & NEAR) d.bslot[kr] = kb++;
                    kr++;
                }
            }
        }
        const int2 lcell = last_cell(d, P, pi);
        for (int j = lcell.x; j < lcell.y; j++) {
            const int h = pair_test(pi, ld32(d.posr2 + j), margin);
            if (h) put(t, i, j, h, -1);
        }
    }
}

// From the scanned counts: row offsets, back rows, every back entry's pair
// into the owner's front row (unordered, with the back entry's place), the
// contact slot of each near back entry, boundary candidates, and per clump the
// members in ascending subsphere order (the order thrust::sort_by_key gives
// reduce_by_key, src/dem_clumpsphere.cu:123-147) with the clump pass's lane
// records.  Contact slots lie in member-slot order: a member's near front
// entries, then its near back entries, and the members of a clump side by
// side, so that the clump pass streams them.
//
// A list longer than its scene's region stops the step before anything current
// is touched (every block finds that for itself; the host grows the regions
// and runs the rebuild again).
static __global__ void __launch_bounds__(SEARCH_THREADS, 8) k_fill(const Dev* __restrict__ dp) {
    constexpr int G = SEARCH_G;
    __shared__ SearchRows sh;
    const Dev& d = *dp;
    if (*d.halt) return;
    const int T = d.plan[PL_T], ns = d.plan[PL_NS], TW = d.plan[PL_TW];
    int over = 0;
    for (int k = threadIdx.x; k < ns; k += SEARCH_THREADS) {
        const int s = d.pscene[k], need = list_need(d, k);
        if (blockIdx.x == 0) d.need[s] = need;
        if (need > d.dyn[s].pcap) {
            over = 1;
            if (blockIdx.x == 0) atomicOr(&d.dyn[s].err, ERR_LIST_OVERFLOW);
        }
    }
    if (__syncthreads_or(over)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *d.halt = 1;   // every later kernel of the step stands still
        return;
    }
    const int g = threadIdx.x % G, grp = threadIdx.x / G;
    const int gshift = (threadIdx.x & 31) & ~(G - 1);
    constexpr unsigned FULL = 0xffffffffu, GM = (1u << G) - 1u;
    const unsigned lt = (1u << g) - 1u;
    const PairList& Nw = d.L[1];
    const int* __restrict__ cnt_f = d.cnt_f;
    const int* __restrict__ cnt_b = d.cnt_b;
    const int* __restrict__ cnt_nf = d.cnt_nf;
    const int* __restrict__ cnt_ns = d.cnt_ns;
    int* __restrict__ fcur = d.fcur;
    int2* __restrict__ tmp = d.tmp;
    for (int b0 = blockIdx.x * SEARCH_GROUPS + (grp & ~3); b0 < T; b0 += gridDim.x * SEARCH_GROUPS) {
        const bool has = b0 + (grp & 3) < T;
        const int t = min(b0 + (grp & 3), T - 1);
        const PlanItem it = plan_item(d, ns, t);
        const int i = it.i, s = it.s, tb = t - i, t0 = d.psub[it.k];
        const ScenePar& P = d.par[s];
        const int base = d.dyn[s].pair_off;
        const int poff = base - cnt_f[t0];
        const int rf = cnt_f[t] + poff, rb = base + cnt_b[t] - cnt_b[t0], nb = cnt_b[t + 1] - cnt_b[t];
        const int nr = base + cnt_nf[t] - cnt_nf[t0], nnf = cnt_nf[t + 1] - cnt_nf[t];
        const int2 ci = d.cm2[i];
        const int s0 = 2 * base + cnt_ns[ci.y + tb] - cnt_ns[t0];
        const int rl = d.rlong[t];
        const bool isl = has && rl == ROW_LONG;
        if (has && g == 0) {
            Nw.row[i + s] = rf;
            Nw.brow[i + s] = rb;
            d.nro[1][i + s] = nr;
            if (i == P.sub_off + P.nsub - 1) {
                Nw.row[i + s + 1] = cnt_f[t + 1] + poff;
                Nw.brow[i + s + 1] = rb + nb;
                d.nro[1][i + s + 1] = nr + nnf;
                d.dyn[s].nbound = d.xcnt[t + 1] - d.xcnt[t0];
            }
            d.nsl[ci.y] = make_int2(s0, cnt_ns[ci.y + tb + 1] - cnt_ns[ci.y + tb]);
            if (d.xcnt[t + 1] - d.xcnt[t]) d.bidx[P.sub_off + d.xcnt[t] - d.xcnt[t0]] = i;
        }
        // a row that is not in the scratch: its candidates once more
        double4 pi = make_double4(0, 0, 0, 0);
        double margin = 0;
        int cand = has && rl != ROW_FACES ? nb : 0, r = 0, kb = s0 + nnf, kr = rb;
        const int* __restrict__ scr = d.scr + (size_t)i * SCR_CAP;
        if (__any_sync(FULL, isl)) {
            pi = ld32(d.posr2 + i);
            margin = near_margin(P);
            const int c = group_rows<false>(d, P, isl && searches(d, P, i), i, pi, g, sh, grp);
            if (isl) cand = c;
        }
        const int most = __reduce_max_sync(FULL, cand);
        for (int k0 = 0; k0 < most; k0 += G) {
            const int k = k0 + g;
            bool hit = k < cand, near = false;
            int v = 0;
            if (hit && !isl) {
                v = scr[k];
                near = v & NEAR;
            } else if (hit) {
                while (sh.row[grp][r].x <= k) r++;
                const int j = k + sh.row[grp][r].y;
                const int h = pair_test(ld32(d.posr2 + j), pi, margin);
                const bool intra = d.cm2[j].x == ci.x;
                hit = h != 0;
                near = h == 2 && !intra;
                v = j | (intra ? INTRA : 0) | (near ? NEAR : 0);
            }
            const unsigned hm = (__ballot_sync(FULL, hit) >> gshift) & GM;
            const unsigned nm = (__ballot_sync(FULL, near) >> gshift) & GM;
            if (hit) {
                const int j = v & SUB_MASK, q = kr + __popc(hm & lt);
                Nw.bnbr[q] = v & ~NEAR;
                tmp[cnt_f[j + tb] + poff + atomicAdd(&fcur[j + tb], 1)] = make_int2(i | (v & ~SUB_MASK), q);
                if (near) d.bslot[q] = kb + __popc(nm & lt);
            }
            kr += __popc(hm);
            kb += __popc(nm);
        }
        if (isl && searches(d, P, i)) {
            const int2 lcell = last_cell(d, P, pi);
            for (int j = lcell.x + g; j < lcell.y; j += G) {
                const int h = pair_test(pi, ld32(d.posr2 + j), margin);
                if (!h) continue;
                const bool intra = d.cm2[j].x == ci.x;
                tmp[rf + atomicAdd(&fcur[t], 1)] =
                    make_int2(j | (intra ? INTRA : 0) | (h == 2 && !intra ? NEAR : 0), -1);
            }
        }
    }
    if (d.plan[PL_FACE]) fill_faces(d);
    // the clump pass's lanes of the rebuilt scenes, a warp per warp of the
    // table: a clump's members change places among its lanes (a thread per
    // clump and a sort in memory: 64 us for the kernel, so 52)
    const int nw = gridDim.x * (SEARCH_THREADS / 32), ln = threadIdx.x & 31;
    for (int u = (blockIdx.x * SEARCH_THREADS + threadIdx.x) / 32; u < TW; u += nw) {
        const int k = plan_find(d.pwarp, ns, u);
        const int s = d.pscene[k];
        const ScenePar& P = d.par[s];
        const int t0 = d.psub[k], tb = t0 - P.sub_off, base = 2 * d.dyn[s].pair_off - cnt_ns[t0];
        const int l = (d.clane[P.clump_off] / 32 + (u - d.pwarp[k])) * 32 + ln;
        int4 ra, rb;
        ld_rec(d.lrec + 2 * (size_t)l, ra, rb);
        const int head = ra.w & 31, nm = ra.w >> 5, c = ra.z;
        const bool mine = c >= 0 && rb.x == s && nm > 0;
        const bool lanes = mine && nm <= 32;
        const int x = lanes ? d.inv[ra.x] : 0;
        int rank = 0;
        const int most = __reduce_max_sync(0xffffffffu, lanes ? nm : 0);
        for (int q = 0; q < most; q++) {
            const int y = __shfl_sync(0xffffffffu, x, head + q);
            if (lanes && q < nm) rank += y < x;
        }
        if (lanes) {
            const int z = cnt_ns[ra.y + tb];
            int4* r = d.lrec + 2 * (size_t)(l - ln + head + rank);   // all lanes have read theirs
            r[0] = make_int4(x, ra.y, c, ra.w);
            r[1] = make_int4(s, base + z, cnt_ns[ra.y + tb + 1] - z, 0);
            d.mo[d.mem_start[c] + rank] = make_int2(x, ra.y);
            // the displacement restarts at zero (src/dem_simulation_clump.cu:172)
            st32(d.cum + ra.y, make_double4(0, 0, 0, 0));
        } else if (mine && ln == 0) {
            // a clump of more than 32 members has the warp to itself
            int2* mo = d.mo;
            const int mb = d.mem_start[c], me = mb + nm;
            for (int m = mb; m < me; m++) {
                st32(d.cum + m, make_double4(0, 0, 0, 0));
                int2 v = mo[m];
                v.x = d.inv[v.x];
                int q = m - 1;
                while (q >= mb && mo[q].x > v.x) { mo[q + 1] = mo[q]; q--; }
                mo[q + 1] = v;
            }
            for (int q = 0; q < 32; q++) {
                const int2 v = mo[mb + q];
                const int z = cnt_ns[v.y + tb];
                d.lrec[2 * (l + q)] = make_int4(v.x, v.y, c, ra.w);
                d.lrec[2 * (l + q) + 1] = make_int4(s, base + z, cnt_ns[v.y + tb + 1] - z, 0);
            }
        }
    }
}

// The front rows in order: 8 lanes per row, each entry's place by counting the
// smaller partners; the half list, the reverse map of CreateContList_cuk
// (src/dem_grid.cu:561-601: the pair of each back entry), and for the near
// pairs the contact pass's work records with the spring histories carried
// over (InheritContHistory_cuk, src/dem_grid.cu:603-647: a pair copies the
// history of the same pair in the current list, negated when the owner
// changed; pairs absent from it start from zero).  Only near pairs can touch
// before the next rebuild, so only they have a history, a touch flag and
// contact slots, and the contact pass visits only them.
//
// A warp takes four rows at a time, 8 lanes each; the near entries, one in
// eight, are put in a queue in shared memory and worked off 32 at a time (done
// in place they ran on two or three lanes of every warp: 65 us at 50,000
// clumps, the queue 57; a row of up to 32 entries in the group's registers,
// its keys compared as they go round, instead of read again for each entry: 50;
// what is left waits on the scattered tmp and records).
constexpr int ROWS_QUEUE = 64;
constexpr int ROWS_HELD = 4;   // entries of a row that a lane of its group holds
template <typename R>
__device__ __forceinline__ void near_record(const Dev& d, int i, int s, int4 e) {
    // e: partner, near pair, listed pair, slot of the back entry (-1: none)
    const int j = e.x, w = e.y;
    const size_t cap = (size_t)d.cap;
    const int* nro = d.nro[0];
    const int2 ci = d.cm2[i], cj = d.cm2[j];
    const int io = d.perm[i], jo = d.perm[j];
    const int oo = min(io, jo), op = max(io, jo);
    const int sf = d.nsl[ci.y].x + (w - d.nro[1][i + s]), sb = e.w;
    const int q0 = nro[oo + s], q1 = nro[oo + s + 1];
    d.rec[1][2 * (size_t)w] = make_int4(i, j, ci.y, cj.y);
    d.rec[1][2 * (size_t)w + 1] = make_int4(ci.x, cj.x, sf, sb);
    d.np[1][w] = e.z;
    // both slots zero until the pair touches
    R4<R>* slots = (R4<R>*)d.slots;
    const R4<R> zero = pack<R>(v3<R>(0, 0, 0), R(0));
    st_pair(slots + 2 * (size_t)sf, zero, zero);
    if (sb >= 0) st_pair(slots + 2 * (size_t)sb, zero, zero);
    uint8_t on = 0;
    // DEMmain::RunSimulation and _Split exchange the history pointers
    // once more after the list build has carried the histories and
    // cleared the other buffer (src/dem_simulation_cylind.cu:141,
    // src/dem_grid.cu:687-749): after a rebuild every pair starts from zero
    if (!(d.par[s].sphere & SPH_RESET)) {
        const R4<R>* Hi = (const R4<R>*)d.H[0];
        R4<R>* Ho = (R4<R>*)d.H[1];
        const int4* orec = d.rec[0];
        const R sign = oo == io ? R(1) : R(-1);
        for (int q = q0; q < q1; q++) {
            if (orec[2 * (size_t)q].y != op) continue;
            if (d.touch[0][q]) {
                R4<R> a, b;
                ld_pair(Hi + 2 * (size_t)q, a, b);
                a.x *= sign; a.y *= sign; a.z *= sign; a.w *= sign;
                b.x *= sign; b.y *= sign; b.z *= sign; b.w *= sign;
                st_pair(Ho + 2 * (size_t)w, a, b);
                ((R*)(Ho + 2 * cap))[w] = sign * ((const R*)(Hi + 2 * cap))[q];
                on = 1;
            }
            break;
        }
    }
    d.touch[1][w] = on;
}

// what the rebuild of every scene built becomes current
static __device__ __noinline__ void commit_pointers(Dev& w) {
#define NBC_SWAP(a, b) { auto tmp_ = w.a; w.a = w.b; w.b = tmp_; }
    NBC_SWAP(posr, posr2) NBC_SWAP(cm, cm2)
    NBC_SWAP(part_fix, part_fix2) NBC_SWAP(level, level2) NBC_SWAP(key, key2)
    NBC_SWAP(bhist, bhist2) NBC_SWAP(bbits, bbits2)
    NBC_SWAP(L[0], L[1]) NBC_SWAP(H[0], H[1]) NBC_SWAP(touch[0], touch[1])
    NBC_SWAP(nro[0], nro[1]) NBC_SWAP(rec[0], rec[1]) NBC_SWAP(np[0], np[1])
#undef NBC_SWAP
}

// (now: the table once more, which the last block of a single scene changes)
template <typename R>
__global__ void __launch_bounds__(SEARCH_THREADS) k_rows(const Dev* __restrict__ dp, Dev* now) {
    constexpr int SL = 8;
    __shared__ int4 s_q[SEARCH_THREADS / 32][ROWS_QUEUE];
    __shared__ int2 s_own[SEARCH_THREADS / 32][ROWS_QUEUE];   // owner, scene
    __shared__ int s_last;
    const Dev& d = *dp;
    if (*d.halt) return;
    const int T = d.plan[PL_T], ns = d.plan[PL_NS];
    const int g = threadIdx.x % SL, ln = threadIdx.x & 31, wp = threadIdx.x / 32;
    const unsigned lt = (1u << ln) - 1u;
    const PairList& Nw = d.L[1];
    const int2* __restrict__ tmp = d.tmp;
    int4* qe = s_q[wp];
    int2* qo = s_own[wp];
    int nq = 0;   // queued entries of the warp
    auto flush = [&](int from) {
        __syncwarp();
        if (from + ln < nq) near_record<R>(d, qo[from + ln].x, qo[from + ln].y, qe[from + ln]);
        __syncwarp();
    };
    // (every lane of a warp takes part in each round: rows past the end are empty)
    const int rpb = SEARCH_THREADS / SL;
    for (int b0 = blockIdx.x * rpb + wp * 4; b0 < T; b0 += gridDim.x * rpb) {
        const int t = b0 + ln / SL;
        int i = 0, s = 0, rf = 0, n = 0, wn = 0;
        if (t < T) {
            const PlanItem it = plan_item(d, ns, t);
            i = it.i;
            s = it.s;
            rf = Nw.row[i + s];
            wn = d.nro[1][i + s];
            n = d.cnt_f[t + 1] - d.cnt_f[t];
            const int hb = d.par[s].bl / 2, nb = d.cnt_b[t + 1] - d.cnt_b[t];
            if (g == 0 && (n > hb || nb > hb)) {
                // the reference's row capacity: back rows, and front rows on one level
                const ScenePar& P = d.par[s];
                int same = n;
                if (P.levels > 1) {
                    const int lv = d.level2[i];
                    const int end = d.cstart[P.cell_off + (lv + 1 < P.levels ? P.loff[lv + 1] : P.cellnum - 1)];
                    same = 0;
                    for (int e = 0; e < n; e++) same += (tmp[rf + e].x & SUB_MASK) < end;
                }
                if (same > hb || nb > hb) atomicOr(&d.dyn[s].err, ERR_ROW_OVERFLOW);
            }
        }
        const int most = __reduce_max_sync(0xffffffffu, n);
        // an entry at its place; near entries to the queue
        auto place = [&](bool has, int2 v, int rank, int nrank) {
            const int p = rf + rank;
            if (has) {
                Nw.nbr[p] = v.x & ~NEAR;
                Nw.own[p] = i;
                if (v.y >= 0) Nw.bpair[v.y] = p;
            }
            const bool near = has && (v.x & NEAR);
            const unsigned nm = __ballot_sync(0xffffffffu, near);
            if (near) {
                const int q = nq + __popc(nm & lt);
                qe[q] = make_int4(v.x & SUB_MASK, wn + nrank, p, v.y >= 0 ? d.bslot[v.y] : -1);
                qo[q] = make_int2(i, s);
            }
            nq += __popc(nm);
            if (nq > ROWS_QUEUE - 32) {
                flush(nq - 32);
                nq -= 32;
            }
        };
        if (most <= SL * ROWS_HELD) {
            // the row in the group's registers: each entry's key (partner, near
            // flag) goes round once and is compared with all of them
            int2 v[ROWS_HELD];
            unsigned key[ROWS_HELD];
            int rank[ROWS_HELD];   // near entries << 16 | entries before
#pragma unroll
            for (int c = 0; c < ROWS_HELD; c++) {
                const bool has = c * SL + g < n;
                v[c] = has ? tmp[rf + c * SL + g] : make_int2(0, -1);
                key[c] = has ? (unsigned)v[c].x << 2 | (v[c].x & NEAR ? 1u : 0u) : 0xffffffffu;
                rank[c] = 0;
            }
#pragma unroll
            for (int b = 0; b < ROWS_HELD; b++) {
                if (b * SL >= most) break;
#pragma unroll
                for (int y = 0; y < SL; y++) {
                    const unsigned w = __shfl_sync(0xffffffffu, key[b], y, SL);
                    const int inc = 1 + (int)((w & 1u) << 16);
#pragma unroll
                    for (int c = 0; c < ROWS_HELD; c++)
                        if (w < key[c]) rank[c] += inc;
                }
            }
#pragma unroll
            for (int c = 0; c < ROWS_HELD; c++)
                if (c * SL < most) place(c * SL + g < n, v[c], rank[c] & 0xffff, rank[c] >> 16);
            continue;
        }
        for (int e0 = 0; e0 < most; e0 += SL) {
            const int e = e0 + g;
            const bool has = e < n;
            const int2 v = has ? tmp[rf + e] : make_int2(0, -1);
            const int j = v.x & SUB_MASK;
            int rank = 0, nrank = 0;
            if (has) {
                for (int y = 0; y < n; y++) {
                    const int w = tmp[rf + y].x;
                    if ((w & SUB_MASK) < j) {
                        rank++;
                        nrank += (w & NEAR) != 0;
                    }
                }
            }
            place(has, v, rank, nrank);
        }
    }
    if (nq > 0) flush(0);
    if (d.S > 1) return;   // k_commit follows
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(d.kc_done, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    // every block is done with the table
    if (threadIdx.x == 0) {
        if (ns) commit_pointers(*now);
    } else if (threadIdx.x == 32) {
        *d.kc_done = 0;
        *d.any_rebuild = 0;
        *d.step_bar = 0ull;
        *d.step_base = 0;
        d.plan[PL_FACE] = 0;
    } else if (threadIdx.x == 64 && ns) {
        SceneDyn& y = d.dyn[0];
        const int np = d.cnt_f[T], nn = d.cnt_nf[T], nb = y.nbound;
        y.npairs = np;
        y.nnear = nn;
        y.nrebuild++;
        y.rebuild = 0;
        d.nprefix[0] = d.bprefix[0] = 0;
        d.nprefix[1] = nn;
        d.bprefix[1] = nb;
    }
}

// Commits a rebuild of several scenes' engine (a single scene's is committed
// by the last block of k_rows).  When every scene was
// rebuilt the gathered buffers, the build list, work records and histories
// become the current ones by exchanging pointers in the table (one thread).
// Otherwise the rebuilt scenes' gathered per-subsphere state, rows, list
// entries, records and histories are copied into the current buffers.  Block 0
// also does the scenes' bookkeeping and the contact and boundary passes' work
// items (near pairs, boundary candidates) as prefixes over the scenes.
template <typename R>
__global__ void __launch_bounds__(SC_THREADS) k_commit(Dev* __restrict__ dp) {
    __shared__ int sh[SC_THREADS / 32];
    const Dev& d = *dp;
    if (*d.halt) return;
    const int ns = d.plan[PL_NS];
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k < ns; k += SC_THREADS) {
            SceneDyn& y = d.dyn[d.pscene[k]];
            const int a = d.psub[k], b = d.psub[k + 1];
            y.npairs = d.cnt_f[b] - d.cnt_f[a];
            y.nnear = d.cnt_nf[b] - d.cnt_nf[a];
            y.nrebuild++;
            y.rebuild = 0;
        }
        if (threadIdx.x == 0) {
            *d.any_rebuild = 0;
            *d.step_bar = 0ull;
            *d.step_base = 0;
            d.plan[PL_FACE] = 0;
        }
        __syncthreads();
        int run = 0, brun = 0;
        for (int b = 0; b < d.S; b += SC_THREADS) {
            const int s = b + threadIdx.x;
            int tot;
            const int ex = block_excl_scan(s < d.S ? d.dyn[s].nnear : 0, sh, tot);
            if (s < d.S) d.nprefix[s] = run + ex;
            run += tot;
            const int bx = block_excl_scan(s < d.S ? d.dyn[s].nbound : 0, sh, tot);
            if (s < d.S) d.bprefix[s] = brun + bx;
            brun += tot;
        }
        if (threadIdx.x == 0) {
            d.nprefix[d.S] = run;
            d.bprefix[d.S] = brun;
        }
    }
    if (ns == d.S) {
        if (blockIdx.x == 0 && threadIdx.x == 0) commit_pointers(*dp);
        return;
    }
    const int T = d.plan[PL_T];
    const size_t N = (size_t)d.N;
    const PairList& Lc = d.L[0];
    const PairList& Nw = d.L[1];
    NBC_GRID_STRIDE(t, T) {
        const PlanItem it = plan_item(d, ns, t);
        const int i = it.i, s = it.s;
        st32(d.posr + i, ld32(d.posr2 + i));
        d.cm[i] = d.cm2[i];
        d.part_fix[i] = d.part_fix2[i];
        d.level[i] = d.level2[i];
        d.key[i] = d.key2[i];
        const uint16_t bits = d.bbits2[i];
        d.bbits[i] = bits;
        const R4<R>* b2 = (const R4<R>*)d.bhist2;
        R4<R>* b1 = (R4<R>*)d.bhist;
        for (int sl = 0; sl < NB_SLOTS; sl++) {
            if (!(bits & (1u << sl))) continue;
            for (int c = 0; c < 3; c++) b1[((size_t)sl * N + i) * 3 + c] = b2[((size_t)sl * N + i) * 3 + c];
        }
        for (int e = 0; e < 2; e++) {   // the row starts, and the end entry of the scene's last row
            if (e == 1 && i != d.par[s].sub_off + d.par[s].nsub - 1) break;
            Lc.row[i + s + e] = Nw.row[i + s + e];
            Lc.brow[i + s + e] = Nw.brow[i + s + e];
            d.nro[0][i + s + e] = d.nro[1][i + s + e];
        }
    }
    const int np = d.cnt_f[T], nn = d.cnt_nf[T];
    const size_t cap = (size_t)d.cap;
    R4<R>* Hc = (R4<R>*)d.H[0];
    const R4<R>* Hn = (const R4<R>*)d.H[1];
    // the lists' entries, then the near pairs' records, of the rebuilt scenes
    NBC_GRID_STRIDE(u, np) {
        int lo = 0, hi = ns - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (d.cnt_f[d.psub[m]] <= u) lo = m;
            else hi = m - 1;
        }
        const int p = d.dyn[d.pscene[lo]].pair_off + (u - d.cnt_f[d.psub[lo]]);
        Lc.nbr[p] = Nw.nbr[p];
        Lc.own[p] = Nw.own[p];
        Lc.bnbr[p] = Nw.bnbr[p];
        Lc.bpair[p] = Nw.bpair[p];
    }
    NBC_GRID_STRIDE(u, nn) {
        int lo = 0, hi = ns - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (d.cnt_nf[d.psub[m]] <= u) lo = m;
            else hi = m - 1;
        }
        const size_t w = (size_t)d.dyn[d.pscene[lo]].pair_off + (u - d.cnt_nf[d.psub[lo]]);
        d.rec[0][2 * w] = d.rec[1][2 * w];
        d.rec[0][2 * w + 1] = d.rec[1][2 * w + 1];
        d.np[0][w] = d.np[1][w];
        const uint8_t f = d.touch[1][w];
        d.touch[0][w] = f;
        if (f) {
            R4<R> a, b;
            ld_pair(Hn + 2 * w, a, b);
            st_pair(Hc + 2 * w, a, b);
            ((R*)(Hc + 2 * cap))[w] = ((const R*)(Hn + 2 * cap))[w];
        }
    }
}

// Moves every scene's list to a new layout of the pair regions (the host
// grows them): entries, back references, and the near pairs' records,
// histories and touch flags.  The contact slots of touching pairs are rewritten
// by the contact pass before they are read; those of the others, which it does
// not write, are zeroed here.  map[s] = (old first slot, new first slot, prefix
// of the pairs over the scenes); d holds the new buffers, o the old ones.
template <typename R>
__global__ void k_relayout(const Dev* __restrict__ dp, Dev o, const int3* __restrict__ map, int total) {
    const Dev& d = *dp;
    const size_t cap = (size_t)d.cap, oc = (size_t)o.cap;
    const R4<R>* Ho = (const R4<R>*)o.H[0];
    R4<R>* Hn = (R4<R>*)d.H[0];
    const PairList& Lc = d.L[0];
    const PairList& ol = o.L[0];
    NBC_GRID_STRIDE(u, total) {
        int lo = 0, hi = d.S - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (map[m].z <= u) lo = m;
            else hi = m - 1;
        }
        const int3 m = map[lo];
        const size_t po = m.x + (u - m.z), pn = m.y + (u - m.z);
        const int delta = m.y - m.x;
        Lc.nbr[pn] = ol.nbr[po];
        Lc.own[pn] = ol.own[po];
        Lc.bnbr[pn] = ol.bnbr[po];
        const int bq = ol.bpair[po];
        Lc.bpair[pn] = bq >= 0 ? bq + delta : bq;
        if (u - m.z >= d.dyn[lo].nnear) continue;
        const int4 a = o.rec[0][2 * po], b = o.rec[0][2 * po + 1];
        d.rec[0][2 * pn] = a;
        const int sf = b.z + 2 * delta, sb = b.w >= 0 ? b.w + 2 * delta : b.w;
        d.rec[0][2 * pn + 1] = make_int4(b.x, b.y, sf, sb);
        d.np[0][pn] = o.np[0][po] + delta;
        const uint8_t f = o.touch[0][po];
        d.touch[0][pn] = f;
        if (f) {
            Hn[2 * pn] = Ho[2 * po];
            Hn[2 * pn + 1] = Ho[2 * po + 1];
            ((R*)(Hn + 2 * cap))[pn] = ((const R*)(Ho + 2 * oc))[po];
        } else {
            R4<R>* slots = (R4<R>*)d.slots;
            const R4<R> zero = pack<R>(v3<R>(0, 0, 0), R(0));
            st_pair(slots + 2 * (size_t)sf, zero, zero);
            if (sb >= 0) st_pair(slots + 2 * (size_t)sb, zero, zero);
        }
    }
}

// the current rows and near rows follow their scene's region: every offset of scene s
// moves by its region's move (the subsphere threads take the row starts and
// the contact slots, one thread per scene the end entry, then the clump pass's lanes)
static __global__ void k_shift_rows(const Dev* __restrict__ dp, const int3* __restrict__ map) {
    const Dev& d = *dp;
    const PairList& Lc = d.L[0];
    NBC_GRID_STRIDE(u, d.N + d.S) {
        int s, r;
        if (u < d.N) {
            s = d.sid[u];
            r = u + s;
            d.nsl[u].x += 2 * (map[s].y - map[s].x);
        } else {
            s = u - d.N;
            r = d.par[s].sub_off + d.par[s].nsub + s;
        }
        const int delta = map[s].y - map[s].x;
        Lc.row[r] += delta;
        Lc.brow[r] += delta;
        d.nro[0][r] += delta;
    }
    NBC_GRID_STRIDE(l, 32 * d.W) {
        int4& b = d.lrec[2 * l + 1];
        b.y += 2 * (map[b.x].y - map[b.x].x);
    }
}

// ===========================================================================
// contact kernel
// ===========================================================================

template <typename R> struct Law {
    double kn_fac, ks_fac, damping;   // stiffness and damping factors (the normal force is FP64)
    R beta, mu, dt;
};

template <typename R> struct LawOut {
    V3<R> Fn, Ft, Mr, Mt;  // normal and tangential force on the body, rolling and twisting moments
    V3<R> hs, ht, hr;      // new tangential, twisting and rolling histories
    R FnL;
};

// The Hertz-Mindlin law with rolling and twisting springs shared by the
// pair, wall and intruder kernels of the reference
// (src/dem_force_clump.cu:66-161, src/dem_force_cube_wall_clump.cu:62-166,
// src/dem_force_penetrator_clump.cu:76-173).  n points from the other body
// toward this body's contact side, Vtot is this body's contact-point velocity
// relative to the other's, Dth = dt (w_this - w_other) for walls and the
// intruder, dt (w_other_side...) as the pair caller passes it.
//
// The normal force Kn Dn n + Cn Vnor is evaluated in FP64 whatever R is: on a
// separating contact its elastic and damping terms nearly cancel (the net
// force of the contact can be a thousandth of either), so rounding them to
// FP32 would leave that contact's force with an error of 1e-4 of itself.  The
// tangential, rolling and twisting parts, the histories and everything after
// run in R.  With R = double every operation is the reference's, in its order.
template <typename R, bool WALL>
__device__ __forceinline__ void hm_law(const Law<R>& L, V3<double> nd, double Dn, V3<double> Vtot, V3<R> Dth,
                                       double Rij, double Mij, R cs_mult, V3<R> H, V3<R> Mr, V3<R> Mt,
                                       LawOut<R>& o) {
    const double sq = sqrt(Rij * Dn);
    const double Kn = L.kn_fac * sq;
    const double Cn = L.damping * sqrt(Kn * Mij);
    const R Ks = (R)(L.ks_fac * sq);
    const R Cs = cs_mult * (R)L.damping * sqrt(Ks * (R)Mij);
    const R br = L.beta * (R)Rij;
    const R Kr = R(0.25) * (R)Kn * br * br;
    const R Cr = R(0.25) * (R)Cn * br * br;
    const R Kt = R(0.50) * Ks * br * br;
    const R Ct = R(0.50) * Cs * br * br;
    const double ERR = dot(nd, Vtot);
    const V3<double> Vnor = ERR * nd;
    const V3<R> Vtan = cvt<R>(Vtot - Vnor);
    const V3<double> Fn = fma2(mul_rn(Kn, Dn), nd, Cn, Vnor);
    const V3<R> n = cvt<R>(nd);
    o.Fn = cvt<R>(Fn);
    o.FnL = (R)len_floor(Fn);
    V3<R> Ft = fma2(-Ks, L.dt * Vtan, Cs, Vtan) + H;
    const R FtL = WALL && sizeof(R) == 8 ? len_floor_yx(Ft) : len_floor(Ft);
    if (FtL > o.FnL * L.mu) {
        Ft = (L.mu * o.FnL * (R(1) / FtL)) * Ft;
        o.hs = Ft;
    } else {
        o.hs = Ft - Cs * Vtan;
    }
    o.Ft = Ft;
    const R DthL = dot(Dth, n);
    const V3<R> DthT = DthL * n;
    const V3<R> DthR = Dth - DthT;
    V3<R> rm = fma1(Kr, DthR, Mr);
    const R rmL = WALL ? len_floor_yx(rm) : len_floor(rm);
    const R rcap = R(0.525) * L.beta * (R)Rij * o.FnL;
    if (rmL > rcap) {
        rm = (rcap * (R(1) / rmL)) * rm;
        o.hr = rm;
    } else {
        o.hr = rm;
        rm = fma1(-(Cr * (R(1) / L.dt)), DthR, rm);
    }
    V3<R> tm = fma1(Kt, DthT, Mt);
    const R tmL = WALL ? len_floor_yx(tm) : len_floor(tm);
    const R tcap = R(0.65) * L.mu * L.beta * (R)Rij * o.FnL;
    if (tmL > tcap) {
        tm = (tcap * (R(1) / tmL)) * tm;
        o.ht = tm;
    } else {
        o.ht = tm;
        tm = fma1(-(Ct * (R(1) / L.dt)), DthT, tm);
    }
    o.Mr = rm;
    o.Mt = tm;
}

// The contact kinematics of a subsphere in FP64 (its clump's velocity and
// angular velocity, its world arm and mass): a bed moving as a whole gives
// touching subspheres nearly equal contact-point velocities, so their
// difference is formed in FP64 before the law rounds anything.  The
// subsphere's own record is one double4 (world arm, mass) written by the
// pose pass; the velocities are read from its clump's records (the values the
// clump pass wrote with the same half-kick), so a clump's velocity is stored
// once rather than once per member.
template <typename R> struct Body {
    double4 p;              // position, radius
    V3<double> v, w, arm;   // clump velocity, clump angular velocity, world arm
    double m;
};

template <typename R>
__device__ __forceinline__ void load_kin(const Dev& d, int2 cm, Body<R>& b) {
    const double4 r = ld32(d.kin + cm.y), v = ld32(d.cvel + cm.x), w = ld32(d.cw + cm.x);
    b.arm = v3(r.x, r.y, r.z);
    b.m = r.w;
    b.v = v3(v.x, v.y, v.z);
    b.w = v3(w.x, w.y, w.z);
}

// The pair law of ContactForce_clump_cuk (src/dem_force_clump.cu:3-163) with
// a in the role of particleI, evaluated once for both bodies of a touching
// pair: the force and torque on a and the torque on b.  Seen from b every
// input of the law is exactly negated (normal, relative velocity, rotation
// increment, negated history), so the law's outputs are negated too: the
// force on b is -fa and its torque uses b's own lever Ab = (rb^2 - ra^2 +
// d^2) / 2d.  Geometry, lever arms and the contact-point velocity are FP64.
// Returns false when the pair does not overlap.
template <typename R>
__device__ __forceinline__ bool pair_contact2(const Law<R>& L, R cohesion, const Body<R>& a, const Body<R>& b,
                                              V3<R> H, V3<R> Mr, V3<R> Mt, V3<R>& fa, V3<R>& ta, V3<R>& tb,
                                              LawOut<R>& o, double& Ap_out, V3<double>& n_out) {
    const double dx = b.p.x - a.p.x, dy = b.p.y - a.p.y, dz = b.p.z - a.p.z;
    const double DistS = fma3(dx, dx, dy, dy, dz, dz);
    const double DistL = sqrt(DistS);
    const double Dn = a.p.w + b.p.w - DistL;
    if (!(Dn > 0.0)) return false;
    const double DistR = 1.0 / DistL;
    const V3<double> nd = v3(DistR * dx, DistR * dy, DistR * dz);
    const double bb = mul_rn(b.p.w, b.p.w);
    const double Ap = mul_rn(0.50 * add_rn(fma_rn(a.p.w, a.p.w, -bb), DistS), DistR);
    const double An = sub_rn(DistL, Ap);
    const double Ab = mul_rn(0.50 * add_rn(fma_rn(-a.p.w, a.p.w, bb), DistS), DistR);
    const double Rij = a.p.w * b.p.w / (a.p.w + b.p.w);
    const double Mij = a.m * b.m / (a.m + b.m);
    const V3<double> ARMa = fma1(Ap, nd, a.arm);
    const V3<double> ARMb = fma1(-An, nd, b.arm);
    const V3<double> Vtot = (b.v - a.v) + (cross(b.w, ARMb) - cross(a.w, ARMa));
    const V3<R> Dth = L.dt * cvt<R>(a.w - b.w);
    hm_law<R, false>(L, nd, Dn, Vtot, Dth, Rij, Mij, R(1), H, Mr, Mt, o);
    const V3<R> n = cvt<R>(nd);
    const R br = L.beta * (R)Rij;
    fa = fma1(cohesion * br * br, n, -o.Fn - o.Ft);
    const V3<R> nxF = cross(n, o.Ft);
    ta = fma1(-(R)Ap, nxF, -o.Mr) - o.Mt;
    tb = fma1(-(R)Ab, nxF, o.Mr) + o.Mt;
    Ap_out = Ap;
    n_out = nd;
    return true;
}

// a wall or intruder contact: normal n (toward the subsphere), lever Ap,
// overlap Dn, wall point RVo relative to the wall centre, wall velocity and
// angular velocity wv, ww (FP64 geometry and velocities, as for pairs)
template <typename R>
__device__ __forceinline__ void boundary_contact(const Law<R>& L, const Body<R>& a, V3<double> nd, double Ap,
                                                 double Dn, V3<double> RVo, V3<double> wv, V3<double> ww,
                                                 double Rij, double Mij, R cs_mult, V3<R> H, V3<R> Mr, V3<R> Mt,
                                                 V3<R>& f, V3<R>& t, LawOut<R>& o, V3<R>& arm_out) {
    const V3<double> Arm = fma1(Ap, nd, -a.arm);
    const V3<double> Vwall = cross(ww, RVo);
    const V3<double> Vtot = (a.v - wv) + (cross(Arm, a.w) - Vwall);
    const V3<R> Dth = L.dt * cvt<R>(a.w - ww);
    hm_law<R, true>(L, nd, Dn, Vtot, Dth, Rij, Mij, cs_mult, H, Mr, Mt, o);
    const V3<R> n = cvt<R>(nd);
    f = o.Fn + o.Ft;
    t = fma1(-(R)Ap, cross(n, o.Ft), -o.Mr) - o.Mt;
    arm_out = cvt<R>(Arm);
}

// pair history layout: R4 (Dv.xyz, Dr.x) at [2q], R4 (Dt.xyz, Dr.y) at
// [2q + 1] (one 32-byte record in FP32), Dr.z as a scalar after the 2*cap R4s
template <typename R>
__device__ __forceinline__ void hist_read(const R4<R>* H, size_t cap, size_t q, V3<R>& hs, V3<R>& ht, V3<R>& hr) {
    R4<R> a, b;
    ld_pair(H + 2 * q, a, b);
    const R c = ((const R*)(H + 2 * cap))[q];
    hs = v3<R>(a.x, a.y, a.z);
    ht = v3<R>(b.x, b.y, b.z);
    hr = v3<R>(a.w, b.w, c);
}
template <typename R>
__device__ __forceinline__ void hist_write(R4<R>* H, size_t cap, size_t q, V3<R> hs, V3<R> ht, V3<R> hr) {
    st_pair(H + 2 * q, pack<R>(hs, hr.x), pack<R>(ht, hr.y));
    ((R*)(H + 2 * cap))[q] = hr.z;
}

constexpr int CT_THREADS = 256;
constexpr int BD_THREADS = 128;

// Walls and intruder, one thread per boundary candidate: the face tests of
// CubeWallInteraction_clump_cuk (src/dem_force_cube_wall_clump.cu:185-298),
// the region tests of CylindWallInteraction_cuk (src/dem_force_cylind_wall.cu:
// 152-237) with clump kinematics, PrePenetrator / GetSphereIntruderContact /
// ForcePene_clump_cuk (src/dem_contact_penetrator.cu:8-84,
// src/dem_sphere_intruder.cuh:20-51, src/dem_force_penetrator_clump.cu:4-182).
// Writes the summed boundary force/torque where some slot is in contact and
// the slot mask; the intruder totals go to fixed-point accumulators.  SPH:
// the build for batches with a sphere-driver scene (ScenePar::sphere); the
// clump path's build carries none of that code.
template <typename R, bool EXPORT, bool SPH>
__device__ __forceinline__ void boundary_one(const Dev& d, const ScenePar& P, int i, int s);

template <typename R, bool EXPORT, bool SPH>
__global__ void __launch_bounds__(BD_THREADS) k_boundary(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    const int S = d.S;
    const int* __restrict__ bpre = d.bprefix;
    const int nb = bpre[S];
    for (int w = blockIdx.x * BD_THREADS + threadIdx.x; w < nb; w += gridDim.x * BD_THREADS) {
        // work item w: boundary candidate w - bprefix[s] of scene s
        const int s = S == 1 ? 0 : plan_find(bpre, S, w);
        const ScenePar& P = d.par[s];
        boundary_one<R, EXPORT, SPH>(d, P, d.bidx[P.sub_off + (w - bpre[s])], s);
    }
}

template <typename R, bool EXPORT, bool SPH>
__device__ __forceinline__ void boundary_one(const Dev& d, const ScenePar& P, int i, int s) {
    const double4 pp = ld32(d.posr + i);   // issued before the scene's flag is known
    const uint16_t bb_old = d.bbits[i];
    if (d.has_stops && d.dyn[s].frozen) return;   // a scene past its stop stands still
    const size_t N = (size_t)d.N;
    const double r = pp.w;
    {
        // conservative early-out: clearly inside every wall and outside the
        // intruder's bounding sphere (margins of 1e-9 relative cover rounding)
        const double ex = pp.x - P.w_c[0], ey = pp.y - P.w_c[1], ez = pp.z - P.w_c[2];
        bool near = false;
        if (P.wall == WALL_CUBE) {
            near = fabs(ex) + r >= P.w_half[0] * (1 - 1e-9) || fabs(ey) + r >= P.w_half[1] * (1 - 1e-9) ||
                   fabs(ez) + r >= P.w_half[2] * (1 - 1e-9);
        } else if (P.wall == WALL_CYL) {
            const double ax = ex * P.cyl_axis[0] + ey * P.cyl_axis[1] + ez * P.cyl_axis[2];
            const double rr = ex * ex + ey * ey + ez * ez - ax * ax;
            const double in = P.cyl_R - r;
            near = fabs(ax) + r >= P.cyl_H * (1 - 1e-9) || in <= 0 || rr >= in * in * (1 - 1e-9);
        }
        if (!near && P.has_intr) {
            const SceneDyn& y = d.dyn[s];
            const double qx = pp.x - y.intr_p[0], qy = pp.y - y.intr_p[1], qz = pp.z - y.intr_p[2];
            const double reach = (P.intr_shape == 1 ? P.intr_R : sqrt(P.intr_R * P.intr_R + P.intr_H * P.intr_H) +
                                  0.80 * P.cell[0] * 1.7320508075688772) + r;
            near = qx * qx + qy * qy + qz * qz <= reach * reach * (1 + 1e-9);
        }
        if (!near) {
            if (bb_old) d.bbits[i] = 0;
            if (EXPORT) {
                R4<R>* xp = (R4<R>*)d.xparts;
                R4<R>* xi = (R4<R>*)d.xintr;
                const R4<R> z = pack<R>(v3<R>(0, 0, 0), R(0));
                for (int c = 2; c < 6; c++) xp[(size_t)c * N + i] = z;
                for (int c = 0; c < 4; c++) xi[(size_t)c * N + i] = z;
            }
            return;
        }
    }
    uint16_t bb_new = 0;
    R4<R>* BH = (R4<R>*)d.bhist;
    V3<R> wF = v3<R>(0, 0, 0), wT = wF, iF = wF, iT = wF;
    Body<R> me;
    bool have_kin = false;
    Law<R> L;
    L.kn_fac = P.kn_fac; L.ks_fac = P.ks_fac; L.damping = P.damping;
    L.beta = (R)P.beta; L.mu = (R)P.mu; L.dt = (R)P.dt;
    const V3<double> RV = v3(pp.x - P.w_c[0], pp.y - P.w_c[1], pp.z - P.w_c[2]);
    // cylinder geometry shared by its three regions
    double ERRc = 0, nrmc = 0;
    V3<double> RVbc = v3(0.0, 0.0, 0.0), RVtc = RVbc, axv = RVbc;
    if (P.wall == WALL_CYL) {
        axv = v3(P.cyl_axis[0], P.cyl_axis[1], P.cyl_axis[2]);
        ERRc = dot(RV, axv);
        RVbc = fma1(-ERRc, axv, RV);
        RVtc = ERRc * axv;
        nrmc = len_floor(RVbc);
    }
    // the slots that may be in contact, then the law slot by slot of the lane's
    // own: lanes on different walls share one evaluation (taking every wall in
    // turn made it three or six)
    unsigned slots = P.has_intr ? 1u << SLOT_INTR : 0u;
    if (P.wall == WALL_CUBE) {
        const double e[3] = {RV.x, RV.y, RV.z};
#pragma unroll
        for (int ax = 0; ax < 3; ax++) {
            const double h = P.w_half[ax];
            if (e[ax] > 0 && e[ax] + r - h > 0) slots |= 1u << (2 * ax);
            if (e[ax] < 0 && e[ax] - r + h < 0) slots |= 2u << (2 * ax);
        }
    } else if (P.wall == WALL_CYL) {
        const double d_cap = fabs(ERRc) - P.cyl_H + r, d_side = nrmc - P.cyl_R + r;
        if (d_cap >= 1e-14 && ERRc < 0) slots |= 1u;
        if (d_cap >= 1e-14 && ERRc > 0) slots |= 2u;
        if (d_side >= 1e-14) slots |= 4u;
    }
#pragma unroll 1
    for (; slots; slots &= slots - 1) {
        const int slot = __ffs(slots) - 1;
        const bool is_intr = slot == SLOT_INTR, is_wall = !is_intr;
        double Apd = 0, Dnd = 0;
        V3<double> nd = v3(0.0, 0.0, 0.0), RVo = nd;
        bool on = false;
        double Rij = r, Mij = 0.0;
        R csm = R(2);
        V3<double> wv = v3(P.w_v[0], P.w_v[1], P.w_v[2]);
        V3<double> ww = v3(P.w_w[0], P.w_w[1], P.w_w[2]);
        if (is_wall && P.wall == WALL_CUBE) {
            const int ax = slot >> 1;
            const bool up = (slot & 1) == 0;
            const double e = (ax == 0 ? RV.x : (ax == 1 ? RV.y : RV.z)), h = P.w_half[ax];
            const double o = (h / fabs(e)) * e;
            RVo = RV;
            if (ax == 0) RVo.x = o; else if (ax == 1) RVo.y = o; else RVo.z = o;
            const double sgn = up ? -1.0 : 1.0;
            if (ax == 0) nd.x = sgn; else if (ax == 1) nd.y = sgn; else nd.z = sgn;
            Apd = dot(RV - RVo, nd);
            Dnd = r - Apd;
            on = Dnd > 0.0;
        } else if (is_wall) {
            RVo = slot < 2 ? fma1(P.cyl_H / fabs(ERRc), RVtc, RVbc) : fma1(P.cyl_R / nrmc, RVbc, RVtc);
            const V3<double> RVn = RV - RVo;
            Dnd = r - len_floor_yx(RVn);
            on = Dnd > 0.0;
            if (on) {
                const double DistL = sqrt(len2_yx(RVn));
                nd = (1.0 / DistL) * RVn;
                Apd = DistL;
            }
        } else {
            const SceneDyn& y = d.dyn[s];
            const V3<double> RI = v3(pp.x - y.intr_p[0], pp.y - y.intr_p[1], pp.z - y.intr_p[2]);
            wv = v3(y.intr_v[0], y.intr_v[1], y.intr_v[2]);
            ww = v3(P.intr_w[0], P.intr_w[1], P.intr_w[2]);
            csm = R(1);
            if (P.intr_shape == 1) {
                const double cd = len_floor(RI);
                if (cd > 1.0e-15) nd = (1.0 / cd) * RI;
                else {
                    V3<double> fb = v3(P.intr_axis[0], P.intr_axis[1], P.intr_axis[2]);
                    double t2 = sqrt(dot(fb, fb));
                    nd = t2 > 1e-20 ? (1.0 / t2) * fb : v3(0.0, 0.0, 0.0);
                    if (len_floor(nd) < 1.0e-15) nd = v3(0.0, 0.0, 1.0);
                }
                RVo = P.intr_R * nd;
                const double gap = cd - P.intr_R;
                Dnd = r - gap;
                Apd = gap;
                on = Dnd > 0.0;
                Rij = r * P.intr_R / (r + P.intr_R);
            } else {
                const double LatDx = P.cell[0];
                const V3<double> pv = v3(P.intr_axis[0], P.intr_axis[1], P.intr_axis[2]);
                const double ERR = dot(RI, pv);
                if (fabs(ERR) < (P.intr_H + 0.80 * LatDx)) {
                    const V3<double> RVb = fma1(-ERR, pv, RI);
                    const double nrm = len_floor(RVb);
                    if (nrm < (P.intr_R + 0.80 * LatDx)) {
                        const V3<double> RVt = ERR * pv;
                        if (fabs(ERR) < P.intr_H) RVo = fma1((1.0 / nrm) * P.intr_R, RVb, RVt);
                        else if (nrm < P.intr_R) RVo = fma1((1.0 / fabs(ERR)) * P.intr_H, RVt, RVb);
                        else RVo = fma2((1.0 / nrm) * P.intr_R, RVb, (1.0 / fabs(ERR)) * P.intr_H, RVt);
                        const V3<double> RVn = RI - RVo;
                        const double DistL = sqrt(dot(RVn, RVn));
                        Dnd = r - DistL;
                        on = Dnd > 0.0;
                        if (on) { nd = (1.0 / DistL) * RVn; Apd = DistL; }
                    }
                }
            }
            if (on && P.intr_wait) atomicCAS(&d.dyn[s].intr_state, 0, 1);
        }
        if (!on) continue;
        if (!have_kin) {
            me.p = pp;
            load_kin<R>(d, d.cm[i], me);
            have_kin = true;
        }
        if (is_intr) Mij = P.intr_motion == 1 ? me.m * P.intr_mass / (me.m + P.intr_mass) : me.m;
        else Mij = me.m;
        V3<R> hs = v3<R>(0, 0, 0), ht = hs, hr = hs;
        const size_t hb = (size_t)slot * 3 * N;
        // the sphere driver's cube wall keeps no history
        const bool memless = SPH && is_wall && P.wall == WALL_CUBE && (P.sphere & SPH_CUBE);
        if (!memless && (bb_old & (1u << slot))) {
            R4<R> a = BH[hb + 3 * i], b = BH[hb + 3 * i + 1], c = BH[hb + 3 * i + 2];
            hs = xyz<R>(a); ht = xyz<R>(b); hr = xyz<R>(c);
        }
        V3<R> f, t, arm;
        LawOut<R> o;
        boundary_contact<R>(L, me, nd, Apd, Dnd, RVo, wv, ww, Rij, Mij, csm, hs, hr, ht,
                            f, t, o, arm);
        if (SPH && memless) {
            // tangential torque only: the moments and the history writes
            // are commented out there (src/dem_force_cube_wall.cu:86-87,137-141)
            t = (-(R)Apd) * cross(cvt<R>(nd), o.Ft);
        } else {
            BH[hb + 3 * i] = pack<R>(o.hs, R(0));
            BH[hb + 3 * i + 1] = pack<R>(o.ht, R(0));
            BH[hb + 3 * i + 2] = pack<R>(o.hr, R(0));
        }
        if (SPH && is_intr && (P.sphere & SPH_KIN)) {
            // the sphere driver's penetrator law adds cohesion
            // (src/dem_force_penetrator.cu:119-123)
            const double cf = ((-P.cohesion) * (P.beta * Rij)) * (P.beta * Rij);
            f = f + cvt<R>(cf * nd);
        }
        bb_new |= (uint16_t)(1u << slot);
        if (is_intr) {
            iF = iF + f;
            iT = iT + t;
            // torque on the intruder about its centre (src/dem_force_penetrator_clump.cu:125,170)
            const V3<R> pt = (-cross(cvt<R>(RVo), f) + o.Mr) + o.Mt;
            long long* fx = (long long*)&d.dyn[s].ifix[0];
            atomicAdd((unsigned long long*)&fx[0], (unsigned long long)llrint((double)f.x * FIX_F));
            atomicAdd((unsigned long long*)&fx[1], (unsigned long long)llrint((double)f.y * FIX_F));
            atomicAdd((unsigned long long*)&fx[2], (unsigned long long)llrint((double)f.z * FIX_F));
            atomicAdd((unsigned long long*)&fx[3], (unsigned long long)llrint((double)pt.x * FIX_T));
            atomicAdd((unsigned long long*)&fx[4], (unsigned long long)llrint((double)pt.y * FIX_T));
            atomicAdd((unsigned long long*)&fx[5], (unsigned long long)llrint((double)pt.z * FIX_T));
            if (EXPORT) {
                R4<R>* xi = (R4<R>*)d.xintr;
                xi[i] = pack<R>(o.Fn, R(0));
                xi[N + i] = pack<R>(o.Ft, R(0));
                xi[2 * N + i] = pack<R>(cross(o.Fn, arm), R(0));
                xi[3 * N + i] = pack<R>((cross(o.Ft, arm) - o.Mr) - o.Mt, R(0));
            }
        } else {
            wF = wF + f;
            wT = wT + t;
        }
    }
    d.bbits[i] = bb_new;
    if (bb_new) {
        R4<R>* fb = (R4<R>*)d.fbnd;
        fb[i] = pack<R>(wF + iF, R(0));
        fb[N + i] = pack<R>(wT + iT, R(0));
        if (SPH && (P.sphere & SPH_KIN) && (bb_new & (1u << SLOT_INTR))) {
            R4<R>* fi = (R4<R>*)d.fint;
            fi[i] = pack<R>(iF, R(0));
            fi[N + i] = pack<R>(iT, R(0));
        }
    }
    if (EXPORT) {
        R4<R>* xp = (R4<R>*)d.xparts;
        xp[2 * N + i] = pack<R>(wF, R(0));
        xp[3 * N + i] = pack<R>(wT, R(0));
        xp[4 * N + i] = pack<R>(iF, R(0));
        xp[5 * N + i] = pack<R>(iT, R(0));
        if (!(bb_new & (1u << SLOT_INTR))) {
            R4<R>* xi = (R4<R>*)d.xintr;
            const R4<R> z = pack<R>(v3<R>(0, 0, 0), R(0));
            xi[i] = z; xi[N + i] = z; xi[2 * N + i] = z; xi[3 * N + i] = z;
        }
    }
}

// Overlap of a listed pair: the reference's test ri + rj - |d| > 0 in FP64
// (src/dem_force_clump.cu:46-50), with the square root taken only when |d|^2
// is within 1e-12 of (ri + rj)^2, so the decision is the reference's exactly.
__device__ __forceinline__ bool overlaps(double4 a, double4 b) {
    const double dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
    const double d2 = dx * dx + dy * dy + dz * dz;
    const double s = a.w + b.w, s2 = s * s;
    if (d2 > s2 * (1.0 + 1e-12)) return false;
    if (d2 < s2 * (1.0 - 1e-12)) return true;
    return a.w + b.w - sqrt(d2) > 0.0;
}

// Pairs, one thread per near pair (grid-stride, so a captured launch covers a
// list that has grown since): the overlap test, and for touching pairs the
// law once (ContactForce_clump_cuk, src/dem_force_clump.cu:3-163, for both
// particles of the pair) and the new spring history.  The force and torque on
// the owner go to one contact slot, those on the partner to another, so the
// clump pass sums every subsphere's contacts from one contiguous range in row
// order; the slots of a pair that does not touch are zero, and are written
// only when it has just come apart (k_rows zeroes them: at the settled beds half
// of the near pairs do not touch, and wrote 64 bytes of zeros each step).  A work record holds
// every index the pair needs, so positions, kinematics, springs and slots are
// one load away from it; the record and touch flag of the next item are
// loaded one ahead, and a pair that touched a step ago loads its kinematics
// and springs beside the positions (FP32 law, 50,000 clumps: 19.4 -> 13.9 us a
// launch; 250,000: the contact phase 129 -> 96 us).  Block 0 marks this step's closing
// half-kick as pending.
constexpr int PR_THREADS = 256;

// resident blocks of k_pairs per SM: the FP64 contact kinematics of two
// bodies need up to 128 registers a thread without spilling
#ifndef NBC_PAIR_MINB
#define NBC_PAIR_MINB 2
#endif
constexpr int CONTACT_LAUNCHES = 2;   // k_pairs and k_boundary

// near pair q with its work record (ra: owner, partner, their member slots; rb:
// their clumps, the slots of the two) and whether it touched a step ago;
// returns whether it touches now
template <typename R, bool EXPORT>
__device__ __forceinline__ uint8_t pair_item(const Dev& d, const ScenePar& P, int4 ra, int4 rb, size_t q, uint8_t was) {
    R4<R>* slots = (R4<R>*)d.slots;
    R4<R>* H = (R4<R>*)d.H[0];
    const size_t cap = (size_t)d.cap;
    Body<R> a, b;
    V3<R> hs = v3<R>(0, 0, 0), ht = hs, hr = hs;
    a.p = ld32(d.posr + ra.x);
    b.p = ld32(d.posr + ra.y);
    // (in FP64 the springs' registers leave no room for that)
    const bool early = sizeof(R) == 4 && was;
    if (early) {
        load_kin<R>(d, make_int2(rb.x, ra.z), a);
        load_kin<R>(d, make_int2(rb.y, ra.w), b);
        hist_read<R>(H, cap, q, hs, ht, hr);
    }
    if (!overlaps(a.p, b.p)) {
        if (was) {
            const R4<R> zero = pack<R>(v3<R>(0, 0, 0), R(0));
            st_pair(slots + 2 * (size_t)rb.z, zero, zero);
            if (rb.w >= 0) st_pair(slots + 2 * (size_t)rb.w, zero, zero);
        }
        return 0;
    }
    if (!early) {
        load_kin<R>(d, make_int2(rb.x, ra.z), a);
        load_kin<R>(d, make_int2(rb.y, ra.w), b);
        if (sizeof(R) == 8 && was) hist_read<R>(H, cap, q, hs, ht, hr);
    }
    Law<R> L;
    L.kn_fac = P.kn_fac; L.ks_fac = P.ks_fac; L.damping = P.damping;
    L.beta = (R)P.beta; L.mu = (R)P.mu; L.dt = (R)P.dt;
    V3<R> fa, ta, tb;
    LawOut<R> o;
    double Ap;
    V3<double> nd;
    pair_contact2<R>(L, (R)P.cohesion, a, b, hs, hr, ht, fa, ta, tb, o, Ap, nd);
    hist_write<R>(H, cap, q, o.hs, o.ht, o.hr);
    st_pair(slots + 2 * (size_t)rb.z, pack<R>(fa, R(0)), pack<R>(ta, R(0)));
    if (rb.w >= 0) st_pair(slots + 2 * (size_t)rb.w, pack<R>(-fa, R(0)), pack<R>(tb, R(0)));
    if (EXPORT) {
        const int p = d.np[0][q];
        R4<R>* xf = (R4<R>*)d.xfcn;
        double4* xc = (double4*)d.xcpt;
        xf[p] = pack<R>(-o.Fn, R(0));
        xc[p] = make_double4(a.p.x + Ap * nd.x, a.p.y + Ap * nd.y, a.p.z + Ap * nd.z, 0.0);
    }
    return 1;
}
template <typename R, bool EXPORT>
__global__ void __launch_bounds__(PR_THREADS, NBC_PAIR_MINB) k_pairs(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *d.post_pending = 1;
    const int S = d.S;
    const int* __restrict__ npre = d.nprefix;
    const int np = npre[S];
    const int4* __restrict__ recs = d.rec[0];
    uint8_t* touch = d.touch[0];
    // work item w: near pair w - nprefix[s] of scene s
    auto fetch = [&](int w, int4& ra, int4& rb, int& s, size_t& q, uint8_t& was) {
        if (w >= np) return false;
        s = S == 1 ? 0 : plan_find(npre, S, w);
        const SceneDyn& ys = d.dyn[s];
        if (d.has_stops && ys.frozen) return false;
        q = (size_t)ys.pair_off + (w - npre[s]);
        ld_rec(recs + 2 * q, ra, rb);
        was = touch[q];
        return true;
    };
    const int stride = gridDim.x * blockDim.x;
    int4 ran = make_int4(0, 0, 0, 0), rbn = ran;
    int sn = 0;
    size_t qn = 0;
    uint8_t wasn = 0;
    bool liven = fetch(blockIdx.x * blockDim.x + threadIdx.x, ran, rbn, sn, qn, wasn);
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < np; w += stride) {
        const int4 ra = ran, rb = rbn;
        const int s = sn;
        const size_t q = qn;
        const uint8_t was = wasn;
        const bool live = liven;
        liven = fetch(w + stride, ran, rbn, sn, qn, wasn);
        if (!live) continue;
        const uint8_t on = pair_item<R, EXPORT>(d, d.par[s], ra, rb, q, was);
        if (on != was) touch[q] = on;
    }
}

// The contact force and torque on subsphere i: its contact slots, then the
// wall and intruder force where a boundary slot is in contact -- the sum the
// clump pass forms, so the per-subsphere totals read back are bitwise the
// ones it integrates.
template <typename R>
__device__ __forceinline__ void contact_sum(const Dev& d, int i, V3<R>& F, V3<R>& T, V3<R>* pairF = nullptr,
                                            V3<R>* pairT = nullptr) {
    const size_t N = (size_t)d.N;
    const int2 sl = d.nsl[d.cm[i].y];
    slot_sum<R>((const R4<R>*)d.slots + 2 * (size_t)sl.x, sl.y, F, T);
    if (pairF) { *pairF = F; *pairT = T; }
    if (d.bbits[i]) {
        const R4<R>* fb = (const R4<R>*)d.fbnd;
        F = F + xyz<R>(fb[i]);
        T = T + xyz<R>(fb[N + i]);
    }
}

// Per subsphere, on request (the force getters and the export step): the
// totals of contact_sum into fsum, the pair part into the export record.
template <typename R, bool EXPORT>
__global__ void __launch_bounds__(CT_THREADS) k_sum(const Dev* __restrict__ dp) {
    const Dev& d = *dp;
    if (*d.halt) return;
    const int i = blockIdx.x * CT_THREADS + threadIdx.x;
    if (i >= d.N) return;
    const size_t N = (size_t)d.N;
    const int s = d.S == 1 ? 0 : d.sid[i];
    if (d.has_stops && d.dyn[s].frozen) return;
    V3<R> F, T, pF, pT;
    contact_sum<R>(d, i, F, T, &pF, &pT);
    if (EXPORT) {
        R4<R>* xp = (R4<R>*)d.xparts;
        xp[i] = pack<R>(pF, R(0));
        xp[N + i] = pack<R>(pT, R(0));
    }
    R4<R>* fo = (R4<R>*)d.fsum;
    fo[i] = pack<R>(F, R(0));
    fo[N + i] = pack<R>(T, R(0));
}

// ===========================================================================
// many steps in one launch
// ===========================================================================

// A grid barrier that also tells whether any block raised `flag`: one 64-bit
// counter, arrivals below, raised flags above, zeroed when a rebuild or a graph
// launch starts it anew (in between, Dev::step_base has the arrivals so far).  The
// wait is bounded (ST_SPIN polls, some seconds); a block that gives up sets
// *fail and *halt and every block leaves at its own limit.  The launch is
// cooperative, so all blocks run at the same time.  Returns 0 or 1, or -1 when
// it gave up; s_out is shared.
constexpr int ST_THREADS = 256;
constexpr int ST_WARPS = ST_THREADS / 32;
constexpr int ST_SCENES = 512;          // scenes whose prefixes fit shared memory
constexpr int ST_SPIN = 1 << 23;
constexpr int ST_MAX_STEPS = 1 << 20;   // steps per launch: the arrivals stay below 2^32

__device__ __forceinline__ int step_barrier(const Dev& d, unsigned target, int flag, int* s_out) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* bar = d.step_bar;
        const unsigned long long add = 1ull | (flag ? 1ull << 32 : 0ull);
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(bar), "l"(add) : "memory");
        unsigned long long v = 0;
        int polls = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
            if ((unsigned)v >= target) break;
            if (++polls > ST_SPIN) {
                atomicExch(d.scan_fail, WAIT_BARRIER);
                atomicExch(d.halt, 1);
                break;
            }
        }
        *s_out = polls > ST_SPIN ? -1 : (int)((v >> 32) != 0);
    }
    __syncthreads();
    return *s_out;
}

// Steps until *loop_left are done, some scene needs a rebuild, or Dev::turn steps
// have been taken: per step the
// clump pass, a grid barrier, pairs and boundary candidates, a grid barrier.
// A step that needs a rebuild leaves the launch after its clump pass (the
// graph's if node runs the rebuild) and the next launch takes up its contact
// pass (*step_phase = 1).  The pointer table and, in a single scene, its
// parameters are kept in shared memory, and so are the work records of a
// warp's first items, which change at rebuilds only: a pass then starts with
// the one load that brings positions, kinematics, springs and slots.
//
// Work items go to the warps block by block (warp w of block b: item
// w gridDim + b), so that a small scene's few warps spread over the SMs.
//
// Bound by latency: at 500 clumps a step is 7,300 cycles of clump pass, 5,400
// of contacts and two barriers of 2,200.  One block of 8 warps per SM with 255
// registers a thread beats 16 warps with 128 and 570 bytes of spilled stack
// (us a step, rebuilds included: 500 clumps 12.9 -> 11.5, 50,000 100 -> 83,
// 250,000 469 -> 432), and one launch per pass (three kernel nodes, fork and
// join, an if and a while node a step: 23.4, 94 and 454 us, 25.8 against 12.4
// for 2,000 spheres in FP64).
template <typename R, bool SPH>
__device__ __noinline__ void boundary_call(const Dev& d, const ScenePar& P, int i, int s) {
    boundary_one<R, false, SPH>(d, P, i, s);
}

template <typename R, bool SPH>
__global__ void __launch_bounds__(ST_THREADS, 1) k_steps(const Dev* __restrict__ dp, cudaGraphConditionalHandle cond,
                                                         cudaGraphConditionalHandle loop) {
    __shared__ Dev s_dev;
    __shared__ ScenePar s_par;
    __shared__ int4 s_lane[ST_THREADS][2], s_pair[ST_THREADS][2];
    __shared__ int s_npre[ST_SCENES + 1], s_bpre[ST_SCENES + 1], s_off[ST_SCENES];
    __shared__ int s_out, s_moved;
    for (int k = threadIdx.x; k < (int)(sizeof(Dev) / sizeof(int)); k += ST_THREADS)
        ((int*)&s_dev)[k] = ((const int*)dp)[k];
    if (threadIdx.x == 0) s_moved = 0;
    __syncthreads();
    const Dev& d = s_dev;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    if (lead) *d.step_runs += 1;
    if (*d.halt) {
        // a rebuild ran out of pair capacity: the host finishes that step
        if (lead) {
            *d.step_phase = 0;
            cudaGraphSetConditional(cond, 0u);
            cudaGraphSetConditional(loop, 0u);
        }
        return;
    }
    const int S = d.S, W = d.W, sw = (S + 31) / 32;
    for (int k = threadIdx.x; S == 1 && k < (int)(sizeof(ScenePar) / sizeof(int)); k += ST_THREADS)
        ((int*)&s_par)[k] = ((const int*)d.par)[k];
    const int lane = threadIdx.x & 31;
    const int gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = gridDim.x * ST_WARPS;
    int L = *d.lstep, post = *d.post_pending, left = *d.loop_left, started = 0;
    const int turn = d.turn;
    bool contact = *d.step_phase != 0;
    const int np = d.nprefix[S], nb = d.bprefix[S];
    const int wp = (np + 31) / 32, wb = (nb + 31) / 32;
    // the warp's first items
    int4 ta = make_int4(-1, 0, -1, 0), tb = make_int4(0, 0, 0, 0);
    if (gw < W) ld_rec(d.lrec + 2 * (size_t)(gw * 32 + lane), ta, tb);
    s_lane[threadIdx.x][0] = ta;
    s_lane[threadIdx.x][1] = tb;
    // the scenes' work items: prefixes, and the first pair slot less the prefix
    const bool tab = S <= ST_SCENES;
    for (int k = threadIdx.x; tab && k <= S; k += ST_THREADS) {
        const int p = d.nprefix[k];
        s_npre[k] = p;
        s_bpre[k] = d.bprefix[k];
        if (k < S) s_off[k] = d.dyn[k].pair_off - p;
    }
    __syncthreads();
    const int* npre = tab ? s_npre : d.nprefix;
    const int* bpre = tab ? s_bpre : d.bprefix;
    // work item w of the contact pass: pair w - nprefix[s] of scene s
    auto pair_of = [&](int w, int& s) {
        s = S == 1 ? 0 : plan_find(npre, S, w);
        return (size_t)((tab ? s_off[s] : d.dyn[s].pair_off - npre[s]) + w);
    };
    int ps = 0;
    size_t pq = 0;
    uint8_t was = 0;
    const bool own = gw * 32 + lane < np;
    if (own) {
        int4 ra, rb;
        pq = pair_of(gw * 32 + lane, ps);
        ld_rec(d.rec[0] + 2 * pq, ra, rb);
        was = d.touch[0][pq];
        s_pair[threadIdx.x][0] = ra;
        s_pair[threadIdx.x][1] = rb;
    }
    const uint8_t was0 = was;
    __syncthreads();
    const ScenePar* par = S == 1 ? &s_par : nullptr;
    unsigned target = *d.step_base;
    int out = 0;
    for (;;) {
        if (!contact) {
            bool moved = false;
            int4 xa = s_lane[threadIdx.x][0], xb = s_lane[threadIdx.x][1];
            for (int w = gw; w < W + sw; w += nw) {
                const int4 ya = xa, yb = xb;
                if (w + nw < W) {   // the next item's
                    ld_rec(d.lrec + 2 * (size_t)((w + nw) * 32 + lane), xa, xb);
                }
                if (w < W) moved |= clump_warp<R, SPH, true>(d, par ? *par : d.par[yb.x], ya, yb, 1, post, L);
                else if ((w - W) * 32 + lane < S) scene_step(d, (w - W) * 32 + lane, 1, post, L);
            }
            if (moved) s_moved = 1;
            L++;
            started++;
            target += gridDim.x;
            __syncthreads();
            out = step_barrier(d, target, s_moved, &s_out);
            if (out) break;
        }
        contact = false;
        int4 xa = s_pair[threadIdx.x][0], xb = s_pair[threadIdx.x][1];
        int xs = ps;
        size_t xq = pq;
        uint8_t xt = was;
        for (int w = gw; w < wp + wb; w += nw) {
            const int4 ra = xa, rb = xb;
            const int s = xs;
            const size_t q = xq;
            const uint8_t t0 = xt;
            if (w + nw < wp && (w + nw) * 32 + lane < np) {   // the next item's
                xq = pair_of((w + nw) * 32 + lane, xs);
                ld_rec(d.rec[0] + 2 * xq, xa, xb);
                xt = d.touch[0][xq];
            }
            if (w < wp) {
                if (w * 32 + lane >= np) continue;
                if (d.has_stops && d.dyn[s].frozen) continue;
                const uint8_t on = pair_item<R, false>(d, par ? *par : d.par[s], ra, rb, q, t0);
                if (w == gw) was = on;   // its flag goes to memory when the launch ends
                else if (on != t0) d.touch[0][q] = on;
            } else {
                const int x = (w - wp) * 32 + lane;
                if (x >= nb) continue;
                const int b = S == 1 ? 0 : plan_find(bpre, S, x);
                const ScenePar& P = par ? *par : d.par[b];
                boundary_call<R, SPH>(d, P, d.bidx[P.sub_off + (x - bpre[b])], b);
            }
        }
        post = 1;
        target += gridDim.x;
        // a raised flag seen here is another block's next clump pass: not yet ours
        out = min(step_barrier(d, target, 0, &s_out), 0);
        left--;
        if (out || left <= 0 || started >= turn) break;
    }
    if (own && was != was0) d.touch[0][pq] = was;
    if (lead) {
        const int reb = out == 1;
        *d.lstep = L;
        *d.hgen += started;
        *d.gstep += started;
        *d.post_pending = post;
        *d.loop_left = left;
        *d.step_phase = reb;
        cudaGraphSetConditional(cond, reb ? 1u : 0u);
        *d.step_base = (int)target;   // (a rebuild starts the barrier anew)
        cudaGraphSetConditional(loop, reb || (out == 0 && left > 0) ? 1u : 0u);
    }
}

// The steps a graph launch takes (the first node of its graph; the count is
// set before each launch) and the barrier's start.
static __global__ void k_loop_init(int* left, int* phase, unsigned long long* bar, int* base, int n) {
    *left = n;
    *phase = 0;
    *bar = 0ull;
    *base = 0;
}

}  // namespace nbc
