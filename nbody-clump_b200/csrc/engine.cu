// engine.cu -- host side of the B200 DEM engine and its C ABI (include/nbc.h).
//
// The Engine owns every device buffer of a batch of scenes, launches the
// kernels of kernels.cuh, captures one step as a CUDA graph whose rebuild
// branch is a conditional node, and converts device data to the reference's
// host layouts on request.  It replaces the host orchestration of
// DEMClumpMain::RunSimulationClump (src/dem_simulation_clump.cu:3-259), which
// synchronises with the device about 30 times per step.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cstdint>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/nbc.h"
#include "kernels.cuh"
#include "engine.h"

namespace nbc {

thread_local std::string g_last_error;

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
// an argument the caller can fix; the C ABI reports it as NBC_ERR_ARG
struct ArgError : std::invalid_argument {
    using std::invalid_argument::invalid_argument;
};

#define CK(call)                                                                             \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            throw CudaError(std::string(#call) + ": " + cudaGetErrorString(e_) + " at " +   \
                            __FILE__ + ":" + std::to_string(__LINE__));                      \
    } while (0)


static inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

// ---------------------------------------------------------------------------
// device memory helper
// ---------------------------------------------------------------------------
// Stream-ordered allocations from the device's default memory pool, kept in
// the pool when freed: creating and destroying engines while others run (a
// request server) neither synchronises the device (as cudaMalloc / cudaFree
// do) nor returns memory to the driver between requests.
struct DevMem {
    std::vector<void*> ptrs;
    double bytes = 0;
    cudaStream_t stream = nullptr;
    template <typename T>
    T* alloc(size_t n) {
        void* p = nullptr;
        size_t b = std::max<size_t>(n, 1) * sizeof(T);
        cudaError_t e = cudaMallocAsync(&p, b, stream);
        if (e != cudaSuccess) throw CudaError(std::string("cudaMalloc ") + std::to_string(b) + ": " + cudaGetErrorString(e));
        CK(cudaMemsetAsync(p, 0, b, stream));
        CK(cudaStreamSynchronize(stream));  // usable from any stream from here on
        ptrs.push_back(p);
        bytes += (double)b;
        return (T*)p;
    }
    void release(void* p, size_t b) {
        for (auto& q : ptrs)
            if (q == p) { cudaFreeAsync(p, stream); q = nullptr; bytes -= (double)b; }
    }
    void free_all() {
        for (void* p : ptrs)
            if (p) cudaFreeAsync(p, stream);
        ptrs.clear();
        if (stream) cudaStreamSynchronize(stream);
    }
    static void keep_pool(int device) {
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
            uint64_t thr = UINT64_MAX;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
        }
    }
};

// Lays buffers out back to back (256-byte aligned) in one slab.  A layout
// function runs twice: with base 0 to size the slab, then with the slab's base.
struct Carver {
    uintptr_t base = 0;
    size_t off = 0;
    template <typename T>
    T* take(size_t n) {
        off = (off + 255) & ~(size_t)255;
        T* p = (T*)(base + off);
        off += std::max<size_t>(n, 1) * sizeof(T);
        return p;
    }
};

// Pinned host words for the engines' asynchronous flag reads, carved from
// pinned blocks shared by all engines of the process (pinned allocation is
// slow): a 16-word slot per engine, returned to a free list.
struct PinnedSlots {
    std::mutex mu;
    std::vector<int*> free_slots;
    int* get() {
        std::lock_guard<std::mutex> lk(mu);
        if (free_slots.empty()) {
            int* blk = nullptr;
            CK(cudaMallocHost(&blk, 4096 * sizeof(int)));
            for (int k = 0; k < 4096; k += 16) free_slots.push_back(blk + k);
        }
        int* p = free_slots.back();
        free_slots.pop_back();
        return p;
    }
    void put(int* p) {
        std::lock_guard<std::mutex> lk(mu);
        free_slots.push_back(p);
    }
};
static PinnedSlots g_pinned;

// A scene's arrays are checked before anything reaches the device: missing
// arrays, non-finite values, non-positive radii, masses and inertias, clump
// ids and grid levels out of range are argument errors (the reference reads
// its inputs unchecked, src/dem_subsphere_io.cu:151-193).
static void validate_scene(const nbc_scene_desc& D, int s) {
    const std::string at = "scene " + std::to_string(s) + ": ";
    if (D.n_sub <= 0 || D.n_clump <= 0 || !D.pos || !D.radius || !D.clump_id || !D.local || !D.mass ||
        !D.clump_pos || !D.clump_vel || !D.clump_quat || !D.clump_angvel || !D.clump_prop)
        throw ArgError(at + "empty or missing arrays");
    if (!(std::isfinite(D.dt) && D.dt > 0)) throw ArgError(at + "time step not positive");
    if (!(std::isfinite(D.thresh) && D.thresh >= 0)) throw ArgError(at + "Thresh negative or not finite");
    if (D.levels > 1 && (!D.level || !D.level_cell)) throw ArgError(at + "grid levels without level arrays");
    auto fin = [](const double* p, int n) {
        for (int k = 0; k < n; k++)
            if (!std::isfinite(p[k])) return false;
        return true;
    };
    for (int i = 0; i < D.n_sub; i++) {
        if (!fin(D.pos + 3 * i, 3) || !fin(D.local + 3 * i, 3))
            throw ArgError(at + "non-finite position at row " + std::to_string(i));
        if (!(std::isfinite(D.radius[i]) && D.radius[i] > 0) || !(std::isfinite(D.mass[i]) && D.mass[i] > 0))
            throw ArgError(at + "radius or mass not positive at row " + std::to_string(i));
        if (D.clump_id[i] < 0 || D.clump_id[i] >= D.n_clump)
            throw ArgError(at + "clump id out of range at row " + std::to_string(i));
        if (D.levels > 1 && (D.level[i] < 0 || D.level[i] >= D.levels))
            throw ArgError(at + "grid level out of range at row " + std::to_string(i));
    }
    for (int k = 0; k < D.n_clump; k++) {
        const double* q = D.clump_quat + 4 * k;
        const double* pr = D.clump_prop + 4 * k;
        if (!fin(D.clump_pos + 3 * k, 3) || !fin(D.clump_vel + 3 * k, 3) || !fin(D.clump_angvel + 3 * k, 3) ||
            !fin(q, 4) || q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3] == 0)
            throw ArgError(at + "non-finite or zero clump state at clump " + std::to_string(k));
        for (int c = 0; c < 4; c++)
            if (!(std::isfinite(pr[c]) && pr[c] > 0))
                throw ArgError(at + "clump inertia or mass not positive at clump " + std::to_string(k));
    }
    for (int l = 0; D.levels > 1 && l < D.levels; l++)
        if (!(std::isfinite(D.level_cell[l]) && D.level_cell[l] > 0))
            throw ArgError(at + "grid cell size not positive on level " + std::to_string(l));
}

// Engines of the process with step launches on their device that nobody has
// waited for yet (see step_grid); one count per device.
static std::atomic<int> g_stepping[64];

template <typename R>
class EngineT final : public EngineBase {
   public:
    EngineT(const std::vector<const nbc_scene_desc*>& sc, const nbc_options& opt, bool shared_gpu)
        : opt_(opt), shared_gpu_(shared_gpu) { setup(sc); }
    ~EngineT() override {
        for (int t = 0; t < 3; t++) {
            if (gexec_[t]) cudaGraphExecDestroy(gexec_[t]);
            if (graph_[t]) cudaGraphDestroy(graph_[t]);
        }
        leave_stepping();
        for (Loop& l : loop_) {
            if (l.exec) cudaGraphExecDestroy(l.exec);
            if (l.graph) cudaGraphDestroy(l.graph);
        }
        for (cudaEvent_t e : ev_) cudaEventDestroy(e);
        for (auto& row : gev_)
            for (cudaEvent_t e : row) if (e) cudaEventDestroy(e);
        if (ev_fork_) cudaEventDestroy(ev_fork_);
        if (ev_join_) cudaEventDestroy(ev_join_);
        mem_.free_all();
        if (stream2_) cudaStreamDestroy(stream2_);
        if (stream_) cudaStreamDestroy(stream_);
        if (hflag_) g_pinned.put(hflag_);
    }

    void step(int n, bool exp) override {
        auto t0 = std::chrono::steady_clock::now();
        int left = n;
        bool checked = false;   // wait_steps has looked for errors
        while (left > 0) {
            if (exp && left == 1) {
                clear_post_done();
                run_step_eager(true);
                checked = false;
                left -= 1;
                continue;
            }
            enqueue(exp ? left - 1 : left);
            left -= wait_steps();
            checked = true;
        }
        if (!checked) {
            CK(cudaStreamSynchronize(stream_));
            check_wait(read_int(h_.scan_fail));
            check_errors();
        }
        last_ms_ = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }

    // Asynchronous stepping: enqueue puts up to n steps on the engine's
    // stream and returns without waiting for them (an engine's first step,
    // and every step without a graph, runs eagerly before it returns);
    // wait_steps waits, finishes a step that a pair-capacity overflow stopped
    // and returns the number of steps done.  A step after an overflow is not
    // done: the caller enqueues the rest again.
    int enqueue(int n) override {
        clear_post_done();
        pend_ = 0;
        pend_eager_ = 0;
        while (n > 0 && (!opt_.use_graph || steps_done_ < 1)) {
            run_step_eager(false);
            pend_eager_++;
            n--;
        }
        if (n <= 0) return pend_eager_;
        cur_ = &loop_[timing_ == 0 ? enter_stepping() : 0];
        if (timing_ == 0 && !cur_->tried) capture_loop(*cur_);
        const Flags f = read_flags();
        pend_before_ = f.v[FL_GSTEP];
        if (timing_ == 0 && cur_->exec) {
            n = std::min(n, ST_MAX_STEPS);
            runs_before_ = f.v[FL_STEP_RUNS];
            launch_loop(n);
        } else {
            if (!gexec_[timing_]) capture(timing_);
            for (int i = 0; i < n; i++) launch_graph();
        }
        pend_ = n;
        return pend_eager_ + n;
    }
    int wait_steps() override {
        int done = pend_eager_;
        if (pend_ > 0) {
            CK(cudaStreamSynchronize(stream_));
            leave_stepping();
            const Flags f = read_flags();
            const int started = f.v[FL_GSTEP] - pend_before_;
            if (timing_ == 0 && cur_->exec) {
                launches_ += 1 + f.v[FL_STEP_RUNS] - runs_before_;   // k_loop_init, k_steps
            } else {
                launches_ += (1LL + CONTACT_LAUNCHES) * started;
            }
            check_wait(f.v[FL_SCAN_FAIL]);
            if (f.v[FL_HALT]) {
                // the last step started stopped at its rebuild: finish it on the host path
                steps_done_ += started - 1;
                recover_halt();
            } else {
                steps_done_ += started;
            }
            done += started;
        } else {
            CK(cudaStreamSynchronize(stream_));
            check_wait(read_int(h_.scan_fail));
        }
        pend_ = pend_eager_ = 0;
        check_errors();
        return done;
    }
    void clear_post_done() {
        if (post_done_) {
            // a sync applied the pending half-kick: the next pass must not repeat it
            CK(cudaMemsetAsync(h_.post_pending, 0, sizeof(int), stream_));
            post_done_ = false;
        }
    }

    void sync() override {
        // apply the pending second half-kick so the state is that of the last step
        int pending = 0;
        CK(cudaStreamSynchronize(stream_));
        copy_(&pending, h_.post_pending, sizeof(int), cudaMemcpyDeviceToHost);
        if (pending && !post_done_) {
            launch_clump(0);
            post_done_ = true;
        }
        CK(cudaStreamSynchronize(stream_));
        refresh_dev();
    }

    // ---- getters ----------------------------------------------------------
    int num_scenes() const override { return S_; }
    void stats(int s, int* steps, int* rebuilds, int* npairs, int* err) override {
        SceneDyn y = read_dyn(s);
        if (steps) *steps = y.step + start_step_[s];
        if (rebuilds) *rebuilds = y.nrebuild;
        if (npairs) *npairs = y.npairs;
        if (err) *err = y.err;
    }
    // near pairs of the current list (the pairs the contact pass visits) and
    // those of them that touched at the last contact pass, over all scenes
    void contact_counts(long long* nnear, long long* ntouch) override {
        refresh_dev();
        std::vector<SceneDyn> y = read_dyn_all();
        long long n = 0, c = 0;
        for (int s = 0; s < S_; s++) {
            std::vector<uint8_t> t(y[s].nnear);
            copy_(t.data(), h_.touch[0] + y[s].pair_off, t.size(), cudaMemcpyDeviceToHost);
            for (uint8_t v : t) c += v != 0;
            n += y[s].nnear;
        }
        if (nnear) *nnear = n;
        if (ntouch) *ntouch = c;
    }
    void get_subspheres(int s, int* fix, int* cid, double* pos, double* rad) override {
        refresh_dev();
        const ScenePar& P = hpar_[s];
        int n = P.nsub, o = P.sub_off;
        if (fix) {
            copy_(fix, h_.part_fix + o, n * sizeof(int), cudaMemcpyDeviceToHost);
        }
        if (cid) {
            k_clump_ids<<<std::min(cdiv(n, 256), sm_count_ * 8), 256, 0, stream_>>>(h_.cm + o, h_.cold, P.clump_off, n,
                                                                                   h_.kA);   // a rebuild's scratch
            CK(cudaGetLastError());
            copy_(cid, h_.kA, n * sizeof(int), cudaMemcpyDeviceToHost);
        }
        if (pos || rad) {
            std::vector<double4> tmp(n);
            copy_(tmp.data(), h_.posr + o, n * sizeof(double4), cudaMemcpyDeviceToHost);
            for (int i = 0; i < n; i++) {
                if (pos) { pos[3 * i] = tmp[i].x; pos[3 * i + 1] = tmp[i].y; pos[3 * i + 2] = tmp[i].z; }
                if (rad) rad[i] = tmp[i].w;
            }
        }
    }
    void get_body(int s, double* local, double* mass) override {
        refresh_dev();
        const ScenePar& P = hpar_[s];
        std::vector<double4> tmp(P.nsub);
        std::vector<int2> cm(P.nsub);
        copy_(tmp.data(), h_.lom + P.sub_off, P.nsub * sizeof(double4), cudaMemcpyDeviceToHost);
        copy_(cm.data(), h_.cm + P.sub_off, P.nsub * sizeof(int2), cudaMemcpyDeviceToHost);
        for (int i = 0; i < P.nsub; i++) {
            const double4& t = tmp[cm[i].y - P.sub_off];   // a scene's member slots are its subsphere range
            if (local) { local[3 * i] = t.x; local[3 * i + 1] = t.y; local[3 * i + 2] = t.z; }
            if (mass) mass[i] = t.w;
        }
    }
    void get_clump_prop(int s, double* prop) override { clumps_out(hpar_[s], {{h_.cprop, prop, 4}}); }
    // clump records of one scene in the caller's order, w doubles each
    struct ClumpOut {
        const double4* src;
        double* dst;
        int w;
    };
    void clumps_out(const ScenePar& P, std::initializer_list<ClumpOut> list) {
        const int n = P.nclump;
        ClumpArrays a{};
        for (const ClumpOut& o : list)
            if (o.dst) {
                a.src[a.n] = o.src;
                a.w[a.n++] = o.w;
            }
        k_clumps_out<<<std::min(cdiv(n, 256), sm_count_ * 8), 256, 0, stream_>>>(a, h_.cold, P.clump_off, n,
                                                                                (double*)h_.stage);
        CK(cudaGetLastError());
        const double* at = (const double*)h_.stage;
        for (const ClumpOut& o : list)
            if (o.dst) {
                copy_(o.dst, at, (size_t)n * o.w * sizeof(double), cudaMemcpyDeviceToHost);
                at += (size_t)n * o.w;
            }
    }
    void get_clumps(int s, double* pos, double* vel, double* quat, double* w, double* f, double* t) override {
        refresh_dev();
        clumps_out(hpar_[s], {{h_.cpos, pos, 3}, {h_.cvel, vel, 3}, {h_.cw, w, 3}, {h_.cF, f, 3}, {h_.cT, t, 3},
                              {h_.cq, quat, 4}});
    }
    void get_sub_forces(int s, double* f, double* t) override {
        refresh_dev();
        launch_sum(false);
        const ScenePar& P = hpar_[s];
        pull_r4(h_.fsum, P.sub_off, P.nsub, f);
        pull_r4((char*)h_.fsum + (size_t)N_ * sizeof(R4<R>), P.sub_off, P.nsub, t);
    }
    void get_force_parts(int s, double* parts) override {
        refresh_dev();
        const ScenePar& P = hpar_[s];
        for (int c = 0; c < 6; c++)
            pull_r4((char*)h_.xparts + (size_t)c * N_ * sizeof(R4<R>), P.sub_off, P.nsub, parts + (size_t)c * P.nsub * 3);
    }
    void get_intruder_diag(int s, double* diag) override {
        refresh_dev();
        const ScenePar& P = hpar_[s];
        for (int c = 0; c < 4; c++)
            pull_r4((char*)h_.xintr + (size_t)c * N_ * sizeof(R4<R>), P.sub_off, P.nsub, diag + (size_t)c * P.nsub * 3);
    }
    void get_pairs(int s, int* np, int* lpa, int* lpb) override {
        refresh_dev();
        SceneDyn y = read_dyn(s);
        const ScenePar& P = hpar_[s];
        int cap_in = *np;
        *np = y.npairs;
        if (!lpa && !lpb) return;
        if (cap_in < y.npairs) throw ArgError("pair buffer too small");
        const PairList& Lc = h_.L[0];
        std::vector<int> own(y.npairs), nbr(y.npairs);
        copy_(own.data(), Lc.own + y.pair_off, y.npairs * sizeof(int), cudaMemcpyDeviceToHost);
        copy_(nbr.data(), Lc.nbr + y.pair_off, y.npairs * sizeof(int), cudaMemcpyDeviceToHost);
        for (int p = 0; p < y.npairs; p++) {
            if (lpa) lpa[p] = own[p] - P.sub_off;
            if (lpb) lpb[p] = (nbr[p] & IDX_MASK) - P.sub_off;
        }
    }
    // the reference's pitched rows (Anei, src/dem_grid.cu:466-552)
    void get_rows(int s, int bl, int* anei, int* ng, int* ni) override {
        RowData rd = pull_rows(s);
        const ScenePar& P = hpar_[s];
        const int n = P.nsub;
        if (anei) std::fill(anei, anei + (size_t)n * bl, -1);
        for (int i = 0; i < n; i++) {
            int nf = rd.row[i + 1] - rd.row[i], nb = rd.brow[i + 1] - rd.brow[i];
            if (ng) ng[i] = nf;
            if (ni) ni[i] = nb;
            if (!anei) continue;
            if (nf > bl / 2 || nb > bl / 2) throw ArgError("row longer than bl/2");
            for (int g = 0; g < nf; g++) anei[(size_t)i * bl + g] = (rd.nbr[rd.row[i] - rd.row[0] + g] & IDX_MASK) - P.sub_off;
            for (int c = 0; c < nb; c++)
                anei[(size_t)i * bl + bl - 1 - c] = (rd.bnbr[rd.brow[i] - rd.brow[0] + c] & IDX_MASK) - P.sub_off;
        }
    }
    // CalFcnChain_cuk (src/dem_force_particle.cu:238-268) on the export data
    void get_chain(int s, int bl, double* fcn, double* cpt) override {
        RowData rd = pull_rows(s);
        const ScenePar& P = hpar_[s];
        const int n = P.nsub;
        SceneDyn y = read_dyn(s);
        std::vector<R4<R>> xf(y.npairs);
        std::vector<double4> xc(y.npairs);
        if (h_.xfcn) {   // zeros where no export step has run
            copy_(xf.data(), (R4<R>*)h_.xfcn + y.pair_off, y.npairs * sizeof(R4<R>), cudaMemcpyDeviceToHost);
            copy_(xc.data(), (double4*)h_.xcpt + y.pair_off, y.npairs * sizeof(double4), cudaMemcpyDeviceToHost);
        }
        std::fill(fcn, fcn + (size_t)n * bl * 3, 0.0);
        std::fill(cpt, cpt + (size_t)n * bl * 3, 0.0);
        const int p0 = rd.row[0];
        for (int i = 0; i < n; i++) {
            for (int g = 0; g < rd.row[i + 1] - rd.row[i]; g++) {
                int p = rd.row[i] - p0 + g;
                double* F = fcn + ((size_t)i * bl + g) * 3;
                double* C = cpt + ((size_t)i * bl + g) * 3;
                if (rd.nbr[p] < 0) continue;
                F[0] = xf[p].x; F[1] = xf[p].y; F[2] = xf[p].z;
                C[0] = xc[p].x; C[1] = xc[p].y; C[2] = xc[p].z;
            }
            for (int c = 0; c < rd.brow[i + 1] - rd.brow[i]; c++) {
                int k = rd.brow[i] - rd.brow[0] + c;
                if (rd.bnbr[k] < 0) continue;
                int p = rd.bpair[k] - y.pair_off;
                double* F = fcn + ((size_t)i * bl + bl - 1 - c) * 3;
                double* C = cpt + ((size_t)i * bl + bl - 1 - c) * 3;
                F[0] = -(double)xf[p].x; F[1] = -(double)xf[p].y; F[2] = -(double)xf[p].z;
                C[0] = xc[p].x; C[1] = xc[p].y; C[2] = xc[p].z;
            }
        }
    }
    // the normal force on the owner of every listed pair, list order (the
    // reference's CacheFcn, src/dem_force_clump.cu:114-116), from the export
    // step; zero for pairs that do not touch
    void get_pair_forces(int s, int* np, double* fcn) override {
        refresh_dev();
        SceneDyn y = read_dyn(s);
        const int cap_in = *np;
        *np = y.npairs;
        if (!fcn) return;
        if (cap_in < y.npairs) throw ArgError("pair buffer too small");
        std::vector<R4<R>> xf(y.npairs);
        if (h_.xfcn) copy_(xf.data(), (R4<R>*)h_.xfcn + y.pair_off, y.npairs * sizeof(R4<R>), cudaMemcpyDeviceToHost);
        for (int p = 0; p < y.npairs; p++) {
            fcn[3 * p] = xf[p].x; fcn[3 * p + 1] = xf[p].y; fcn[3 * p + 2] = xf[p].z;
        }
    }
    void get_intruder(int s, double* pos, double* vel, double* reac, double* tq, int* state) override {
        SceneDyn y = read_dyn(s);
        for (int c = 0; c < 3; c++) {
            if (pos) pos[c] = y.intr_p[c];
            if (vel) vel[c] = y.intr_v[c];
            if (reac) reac[c] = y.reaction[c];
            if (tq) tq[c] = y.reaction_t[c];
        }
        if (state) *state = y.intr_state;
    }
    void get_intruder_history(int s, int count, double* out) override {
        SceneDyn y = read_dyn(s);
        if (count > ring_len_) throw ArgError("history longer than the ring");
        std::vector<double> ring((size_t)ring_len_ * 6);
        copy_(ring.data(), h_.ring + (size_t)s * ring_len_ * 6, ring.size() * sizeof(double),
                      cudaMemcpyDeviceToHost);
        for (int c = 0; c < count; c++) {
            int st = y.step - count + c;
            if (st < 0) { for (int q = 0; q < 6; q++) out[c * 6 + q] = 0; continue; }
            int slot = st % ring_len_;
            for (int q = 0; q < 6; q++) out[c * 6 + q] = ring[(size_t)slot * 6 + q];
        }
    }
    void timing_enable(int level) override {
        CK(cudaStreamSynchronize(stream_));
        timing_ = level <= 0 ? 0 : (level == 1 ? 1 : 2);
        for (double& v : t_phase_ms_) v = 0;
        t_contact_n_ = 0;
        launches_ = 0;
        rebuilds_at_enable_ = total_rebuilds();
        ev_used_ = 0;
    }
    void timing_read(double* ms, int* nc, long long* nk, int* nr) override {
        CK(cudaStreamSynchronize(stream_));
        harvest_events();
        if (ms) *ms = t_phase_ms_[PH_CONTACT];
        if (nc) *nc = t_contact_n_;
        if (nk) *nk = launches_ + (long long)(total_rebuilds() - rebuilds_at_enable_) * rebuild_launches();
        if (nr) *nr = total_rebuilds() - rebuilds_at_enable_;
    }
    void timing_phases(double* ms) override {
        CK(cudaStreamSynchronize(stream_));
        harvest_events();
        for (int k = 0; k < NPH; k++) ms[k] = t_contact_n_ ? t_phase_ms_[k] / t_contact_n_ : 0.0;
    }
    // scene s stands still after nsteps steps counted from the engine's creation
    void set_stop(int s, int nsteps) override {
        if (s < 0 || s >= S_) throw ArgError("scene index out of range");
        if (nsteps < 0) throw ArgError("scene step count is negative");
        const int started = read_int(h_.lstep);
        if (nsteps != 0 && nsteps < started)
            throw ArgError("scene " + std::to_string(s) + " has started " + std::to_string(started) + " steps already");
        SceneDyn y = read_dyn(s);
        y.stop = nsteps;
        copy_(h_.dyn + s, &y, sizeof(SceneDyn), cudaMemcpyHostToDevice);
        if (nsteps && !h_.has_stops) {
            refresh_dev();
            h_.has_stops = 1;
            push_dev();
        }
    }
    // ---- exact checkpoint -------------------------------------------------
    // The state a step leaves for the next one, after nbc_sync (the pending
    // half-kick applied): every scene's bookkeeping (SceneDyn: steps, intruder
    // state, pair region, step limit), the history generation and step
    // counters, every subsphere in the current sort order (position and
    // radius, body offset and mass, displacement since the last rebuild,
    // clump, original index, grid level, cell key, contact kinematics, wall
    // and intruder spring histories and their contact bits, boundary
    // candidates), every clump's state and member list, and each scene's
    // pair region: the current half list with its back references, spring
    // histories and touch flags, the near rows and their contact slots, and
    // the intruder force ring.  Rebuild scratch is not saved: a rebuild
    // writes it before reading it.  Loading this into an engine made from
    // the same scenes and options and stepping on gives bitwise the run that
    // never stopped (the reference restarts from StartStep, src/world.par:28
    // and src/dem_simulation_clump.cu:110, with its spring histories lost).
    struct CkHeader {
        char magic[8];
        int version, S, N, K, cells, real_bytes, steps_done, hgen, gstep, lstep, ring_len;
        long long total_cap;
    };
    std::vector<char> checkpoint_save() override {
        if (steps_done_ < 1) throw StateError("checkpoint before the first step (there is no list yet)");
        sync();
        refresh_dev();
        CkHeader hd{};
        memcpy(hd.magic, "NBCCKPT", 8);
        hd.version = 1;
        hd.S = S_; hd.N = N_; hd.K = K_; hd.cells = h_.cells;
        hd.real_bytes = (int)sizeof(R);
        hd.steps_done = steps_done_;
        hd.hgen = read_int(h_.hgen);
        hd.gstep = read_int(h_.gstep);
        hd.lstep = read_int(h_.lstep);
        hd.ring_len = ring_len_;
        hd.total_cap = h_.cap;
        // what the file holds per subsphere, clump and pair, in one allocation
        size_t pairs = 0, near = 0;
        for (const SceneDyn& y : read_dyn_all()) { pairs += y.npairs; near += y.nnear; }
        std::vector<char> out;
        out.reserve(sizeof(hd) + S_ * (sizeof(SceneDyn) + (size_t)ring_len_ * 48 + 64) + (size_t)K_ * 264 +
                    (size_t)N_ * (176 + (NB_SLOTS * 3 + 4) * sizeof(R4<R>)) + pairs * (26 + hist_bytes(1)) +
                    near * (20 + 4 * sizeof(R4<R>)) + 4096);
        out.assign((const char*)&hd, (const char*)&hd + sizeof(hd));
        ck_blocks(out, nullptr, 0, 0, hd);
        return out;
    }
    void checkpoint_load(const char* data, size_t bytes) override {
        if (bytes < sizeof(CkHeader)) throw ArgError("checkpoint too short");
        CkHeader hd;
        memcpy(&hd, data, sizeof(hd));
        if (memcmp(hd.magic, "NBCCKPT", 8) != 0 || hd.version != 1) throw ArgError("not an engine checkpoint");
        if (hd.S != S_ || hd.N != N_ || hd.K != K_ || hd.cells != h_.cells || hd.ring_len != ring_len_)
            throw ArgError("checkpoint of different scenes");
        if (hd.real_bytes != (int)sizeof(R)) throw ArgError("checkpoint of the other precision");
        if (bytes < sizeof(hd) + S_ * sizeof(SceneDyn)) throw ArgError("checkpoint too short");
        CK(cudaStreamSynchronize(stream_));
        // pair regions as saved (their sizes are in the saved SceneDyn)
        refresh_dev();
        mem_.release(pslab_, pslab_bytes_);
        alloc_pairs(std::max<long long>(hd.total_cap, 1));
        push_dev();
        std::vector<char> none;
        ck_blocks(none, data, bytes, sizeof(hd), hd);
        steps_done_ = hd.steps_done;
        first_list_ = false;
        post_done_ = false;
        pend_ = pend_eager_ = 0;
        bool stops = false;
        for (const SceneDyn& v : read_dyn_all()) stops |= v.stop != 0;
        if (stops && !h_.has_stops) {
            h_.has_stops = 1;
            push_dev();
        }
        CK(cudaStreamSynchronize(stream_));
    }
    // Writes (src == nullptr: appends to out) or reads (from src at offset
    // off) the checkpoint's blocks in one fixed order.  The file holds clumps
    // in the caller's order and what the engine keeps per member slot in
    // subsphere order, so it does not depend on the engine's own order.
    void ck_blocks(std::vector<char>& out, const char* src, size_t size, size_t off, const CkHeader& hd) {
        const size_t N = N_;
        auto blk = [&](void* dev, size_t n) {
            if (!n) return;
            if (!src) {
                const size_t at = out.size();
                out.resize(at + n);
                copy_(out.data() + at, dev, n, cudaMemcpyDeviceToHost);
            } else {
                if (off + n > size) throw ArgError("checkpoint truncated");
                copy_(dev, src + off, n, cudaMemcpyHostToDevice);
                off += n;
            }
        };
        // the same for a block that the host holds
        auto hblk = [&](void* host, size_t n) {
            if (!n) return;
            if (!src) {
                const size_t at = out.size();
                out.resize(at + n);
                memcpy(out.data() + at, host, n);
            } else {
                if (off + n > size) throw ArgError("checkpoint truncated");
                memcpy(host, src + off, n);
                off += n;
            }
        };
        // an array of the clumps, in the caller's order in the file
        auto cblk = [&](double4* dev) {
            std::vector<double4> own(K_), file(K_);
            if (!src) {
                copy_(own.data(), dev, K_ * sizeof(double4), cudaMemcpyDeviceToHost);
                for (int s = 0; s < S_; s++)
                    for (int c = hpar_[s].clump_off; c < hpar_[s].clump_off + hpar_[s].nclump; c++)
                        file[hpar_[s].clump_off + cold_[c]] = own[c];
            }
            hblk(file.data(), K_ * sizeof(double4));
            if (src) {
                for (int s = 0; s < S_; s++)
                    for (int c = hpar_[s].clump_off; c < hpar_[s].clump_off + hpar_[s].nclump; c++)
                        own[c] = file[hpar_[s].clump_off + cold_[c]];
                copy_(dev, own.data(), K_ * sizeof(double4), cudaMemcpyHostToDevice);
            }
        };
        // scene bookkeeping first (its pair regions size the rest)
        blk(h_.dyn, S_ * sizeof(SceneDyn));
        std::vector<SceneDyn> y = read_dyn_all();
        // counters; the pending half-kick was applied by sync, so the next
        // step must not repeat it (post_pending saved as 0)
        int flags[4] = {hd.hgen, hd.gstep, hd.lstep, 0};
        if (!src) {
            const size_t at = out.size();
            out.resize(at + sizeof(flags));
            memcpy(out.data() + at, flags, sizeof(flags));
        } else {
            if (off + sizeof(flags) > size) throw ArgError("checkpoint truncated");
            memcpy(flags, src + off, sizeof(flags));
            off += sizeof(flags);
            copy_(h_.hgen, &flags[0], sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.gstep, &flags[1], sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.lstep, &flags[2], sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.post_pending, &flags[3], sizeof(int), cudaMemcpyHostToDevice);
            int zero = 0;
            copy_(h_.any_rebuild, &zero, sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.halt, &zero, sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.kc_done, &zero, sizeof(int), cudaMemcpyHostToDevice);
        }
        // subspheres, current sort order
        blk(h_.posr, N * sizeof(double4));
        std::vector<int2> cm(N);
        std::vector<double4> slot[3], file[3];   // lom, cum, kin by member slot and by subsphere
        std::vector<int> cid(N), fix(N);
        double4* slot_dev[3] = {h_.lom, h_.cum, h_.kin};
        for (int a = 0; a < 3; a++) { slot[a].resize(N); file[a].resize(N); }
        if (!src) {
            copy_(cm.data(), h_.cm, N * sizeof(int2), cudaMemcpyDeviceToHost);
            copy_(fix.data(), h_.part_fix, N * sizeof(int), cudaMemcpyDeviceToHost);
            for (int a = 0; a < 3; a++) copy_(slot[a].data(), slot_dev[a], N * sizeof(double4), cudaMemcpyDeviceToHost);
            for (int s = 0; s < S_; s++)
                for (int i = hpar_[s].sub_off; i < hpar_[s].sub_off + hpar_[s].nsub; i++) {
                    cid[i] = hpar_[s].clump_off + cold_[cm[i].x];
                    for (int a = 0; a < 3; a++) file[a][i] = slot[a][cm[i].y];
                }
        }
        hblk(file[0].data(), N * sizeof(double4));
        hblk(file[1].data(), N * sizeof(double4));
        hblk(cid.data(), N * sizeof(int));
        hblk(fix.data(), N * sizeof(int));
        blk(h_.level, N * sizeof(int));
        blk(h_.key, N * sizeof(int));
        hblk(file[2].data(), N * sizeof(double4));
        if (src) {
            for (int s = 0; s < S_; s++)
                for (int i = hpar_[s].sub_off; i < hpar_[s].sub_off + hpar_[s].nsub; i++) {
                    if (fix[i] < 0 || fix[i] >= hpar_[s].nsub) throw ArgError("checkpoint of different scenes");
                    const int m = mrow_[hpar_[s].sub_off + fix[i]];
                    cm[i] = make_int2(mcl_[m], m);
                    cid[i] = hpar_[s].clump_off + cold_[mcl_[m]];
                    for (int a = 0; a < 3; a++) slot[a][m] = file[a][i];
                }
            copy_(h_.cm, cm.data(), N * sizeof(int2), cudaMemcpyHostToDevice);
            copy_(h_.part_fix, fix.data(), N * sizeof(int), cudaMemcpyHostToDevice);
            for (int a = 0; a < 3; a++) copy_(slot_dev[a], slot[a].data(), N * sizeof(double4), cudaMemcpyHostToDevice);
        }
        blk(h_.bhist, (size_t)NB_SLOTS * 3 * N * sizeof(R4<R>));
        blk(h_.bbits, N * sizeof(uint16_t));
        blk(h_.fbnd, 2 * N * sizeof(R4<R>));
        if (h_.fint) blk(h_.fint, 2 * N * sizeof(R4<R>));
        blk(h_.bidx, N * sizeof(int));
        // clumps
        for (double4* a : {h_.cpos, h_.cvel, h_.cw, h_.cq, h_.cprop, h_.cinv}) cblk(a);
        // the member lists, by the caller's clump number (follow from the
        // subspheres' clumps, so a load makes them from those)
        std::vector<int> fcl(N), fst(K_ + 1, 0), fidx(N);
        for (size_t i = 0; i < N; i++) fst[cid[i] + 1]++;
        for (int k = 0; k < K_; k++) fst[k + 1] += fst[k];
        {
            std::vector<int> cur(fst.begin(), fst.end() - 1);
            for (size_t i = 0; i < N; i++) fidx[cur[cid[i]]++] = (int)i;
        }
        for (int k = 0; k < K_; k++)
            for (int m = fst[k]; m < fst[k + 1]; m++) fcl[m] = k;
        hblk(fcl.data(), N * sizeof(int));
        cblk(h_.cF);
        cblk(h_.cT);
        hblk(fst.data(), (K_ + 1) * sizeof(int));
        hblk(fidx.data(), N * sizeof(int));
        if (src) {
            std::vector<int> cur(mstart_.begin(), mstart_.end() - 1);
            std::vector<int2> mo(N);
            for (size_t i = 0; i < N; i++) mo[cur[cm[i].x]++] = make_int2((int)i, cm[i].y);
            copy_(h_.mo, mo.data(), N * sizeof(int2), cudaMemcpyHostToDevice);
        }
        // rows and work-item prefixes
        blk(h_.L[0].row, (N + S_) * sizeof(int));
        blk(h_.L[0].brow, (N + S_) * sizeof(int));
        // near rows in the file: offsets of each subsphere's near front and
        // near back entries, the contact slots in that order
        std::vector<int2> nrb(N + S_);
        std::vector<int> nro(N + S_);
        std::vector<int2> nsl(N);
        if (!src) {
            copy_(nro.data(), h_.nro[0], (N + S_) * sizeof(int), cudaMemcpyDeviceToHost);
            copy_(nsl.data(), h_.nsl, N * sizeof(int2), cudaMemcpyDeviceToHost);
            for (int s = 0; s < S_; s++) {
                int back = y[s].pair_off;
                const int e = hpar_[s].sub_off + hpar_[s].nsub;
                for (int i = hpar_[s].sub_off; i < e; i++) {
                    nrb[i + s] = make_int2(nro[i + s], back);
                    back += nsl[cm[i].y].y - (nro[i + s + 1] - nro[i + s]);
                }
                nrb[e + s] = make_int2(nro[e + s], back);
            }
        }
        hblk(nrb.data(), (N + S_) * sizeof(int2));
        if (src) {
            for (int s = 0; s < S_; s++) {
                int at = 2 * y[s].pair_off;
                const int o = hpar_[s].sub_off, e = o + hpar_[s].nsub;
                for (int i = o; i <= e; i++) nro[i + s] = nrb[i + s].x;
                std::vector<int> row(hpar_[s].nsub);   // subsphere of each member slot
                for (int i = o; i < e; i++) row[cm[i].y - o] = i;
                for (int m = o; m < e; m++) {
                    const int2 a = nrb[row[m - o] + s], b = nrb[row[m - o] + s + 1];
                    nsl[m] = make_int2(at, (b.x - a.x) + (b.y - a.y));
                    at += nsl[m].y;
                    if (nsl[m].y < 0 || at > 2 * (y[s].pair_off + y[s].pcap)) throw ArgError("checkpoint of different scenes");
                }
            }
            copy_(h_.nro[0], nro.data(), (N + S_) * sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.nsl, nsl.data(), N * sizeof(int2), cudaMemcpyHostToDevice);
            std::vector<int4> lr(2 * 32 * (size_t)h_.W);
            copy_(lr.data(), h_.lrec, lr.size() * sizeof(int4), cudaMemcpyDeviceToHost);
            std::vector<int2> mo(N);
            copy_(mo.data(), h_.mo, N * sizeof(int2), cudaMemcpyDeviceToHost);
            for (int k = 0; k < K_; k++)
                for (int m = mstart_[k]; m < std::min(mstart_[k + 1], mstart_[k] + 32); m++) {
                    int4* r = &lr[2 * (size_t)(clane_[k] + m - mstart_[k])];
                    r[0].x = mo[m].x; r[0].y = mo[m].y;
                    r[1].y = nsl[mo[m].y].x; r[1].z = nsl[mo[m].y].y;
                }
            copy_(h_.lrec, lr.data(), lr.size() * sizeof(int4), cudaMemcpyHostToDevice);
        }
        blk(h_.nprefix, (S_ + 1) * sizeof(int));
        blk(h_.bprefix, (S_ + 1) * sizeof(int));
        blk(h_.ring, (size_t)S_ * ring_len_ * 6 * sizeof(double));
        // each scene's pair region; springs, touch and near flags per listed
        // pair in the file, per near pair here
        const size_t cap = h_.cap;
        for (int s = 0; s < S_; s++) {
            const size_t o = y[s].pair_off, np = y[s].npairs, nn = y[s].nnear;
            if (src && (np > (size_t)y[s].pcap || nn > np || o + np > cap)) throw ArgError("checkpoint of different scenes");
            blk(h_.L[0].nbr + o, np * sizeof(int));
            blk(h_.L[0].own + o, np * sizeof(int));
            blk(h_.L[0].bnbr + o, np * sizeof(int));
            blk(h_.L[0].bpair + o, np * sizeof(int));
            std::vector<R4<R>> hf(2 * np), hn(2 * nn), fs(2 * nn), bs(2 * nn), sl(4 * nn);
            std::vector<R> zf(np), zn(nn);
            std::vector<uint8_t> tf(np), tn(nn), nf(np);
            std::vector<int> pos(np, -1), nbq(nn), pr(nn);
            std::vector<int4> nfr(nn), rec(2 * nn);
            R4<R>* H = (R4<R>*)h_.H[0];
            R4<R>* S = (R4<R>*)h_.slots;
            if (!src) {
                std::vector<int> brow(hpar_[s].nsub + 1), bpair(np);
                copy_(hn.data(), H + 2 * o, 2 * nn * sizeof(R4<R>), cudaMemcpyDeviceToHost);
                copy_(zn.data(), (R*)(H + 2 * cap) + o, nn * sizeof(R), cudaMemcpyDeviceToHost);
                copy_(tn.data(), h_.touch[0] + o, nn, cudaMemcpyDeviceToHost);
                copy_(pr.data(), h_.np[0] + o, nn * sizeof(int), cudaMemcpyDeviceToHost);
                copy_(rec.data(), h_.rec[0] + 2 * o, 2 * nn * sizeof(int4), cudaMemcpyDeviceToHost);
                copy_(sl.data(), S + 4 * o, 4 * nn * sizeof(R4<R>), cudaMemcpyDeviceToHost);
                copy_(brow.data(), h_.L[0].brow + hpar_[s].sub_off + s, brow.size() * sizeof(int), cudaMemcpyDeviceToHost);
                copy_(bpair.data(), h_.L[0].bpair + o, np * sizeof(int), cudaMemcpyDeviceToHost);
                for (size_t w = 0; w < nn; w++) nf[pr[w] - o] = 1;
                size_t e = 0;
                for (int k = brow.front(); k < brow.back(); k++) {
                    const int q = bpair[k - o];
                    if (q < 0 || !nf[q - o] || e >= nn) continue;
                    pos[q - o] = (int)(o + e);
                    nbq[e++] = q;
                }
                for (size_t w = 0; w < nn; w++) {
                    const size_t p = pr[w] - o;
                    const int4 a = rec[2 * w], b = rec[2 * w + 1];
                    nfr[w] = make_int4(pr[w], a.y, a.x, pos[p]);
                    tf[p] = tn[w];
                    if (tn[w]) { hf[2 * p] = hn[2 * w]; hf[2 * p + 1] = hn[2 * w + 1]; zf[p] = zn[w]; }
                    for (int c = 0; c < 2; c++) {
                        fs[2 * w + c] = sl[2 * (b.z - 2 * o) + c];
                        if (pos[p] >= 0) bs[2 * (pos[p] - o) + c] = sl[2 * (b.w - 2 * o) + c];
                    }
                }
            }
            hblk(hf.data(), 2 * np * sizeof(R4<R>));
            hblk(zf.data(), np * sizeof(R));
            hblk(tf.data(), np);
            hblk(nf.data(), np);
            hblk(pos.data(), np * sizeof(int));
            hblk(nfr.data(), nn * sizeof(int4));
            hblk(nbq.data(), nn * sizeof(int));
            hblk(fs.data(), 2 * nn * sizeof(R4<R>));
            hblk(bs.data(), 2 * nn * sizeof(R4<R>));
            if (src) {
                const int lo = hpar_[s].sub_off, hi = lo + hpar_[s].nsub;
                for (size_t w = 0; w < nn; w++) {
                    const int4 v = nfr[w];
                    const size_t p = (size_t)((long long)v.x - (long long)o);
                    if (p >= np || v.y < lo || v.y >= hi || v.z < lo || v.z >= hi) throw ArgError("checkpoint of different scenes");
                    const int2 ci = cm[v.z], cj = cm[v.y];
                    const int2 ri = nrb[v.z + s], rj = nrb[v.y + s], rj1 = nrb[v.y + s + 1];
                    const int sf = nsl[ci.y].x + (int)(o + w) - ri.x;
                    // the partner's near back entry, behind its near front entries (-1: it has none)
                    const int e = v.w, own = e >= rj.y && e < rj1.y && nbq[e - o] == v.x;
                    const int sb = own ? nsl[cj.y].x + (rj1.x - rj.x) + (e - rj.y) : -1;
                    if (sf < 2 * (int)o || sf >= 2 * (int)(o + nn) || sb >= 2 * (int)(o + nn))
                        throw ArgError("checkpoint of different scenes");
                    rec[2 * w] = make_int4(v.z, v.y, ci.y, cj.y);
                    rec[2 * w + 1] = make_int4(ci.x, cj.x, sf, sb);
                    pr[w] = v.x;
                    tn[w] = tf[p];
                    hn[2 * w] = hf[2 * p]; hn[2 * w + 1] = hf[2 * p + 1]; zn[w] = zf[p];
                    for (int c = 0; c < 2; c++) {
                        sl[2 * (sf - 2 * o) + c] = fs[2 * w + c];
                        if (sb >= 0) sl[2 * (sb - 2 * o) + c] = bs[2 * (e - o) + c];
                    }
                }
                copy_(H + 2 * o, hn.data(), 2 * nn * sizeof(R4<R>), cudaMemcpyHostToDevice);
                copy_((R*)(H + 2 * cap) + o, zn.data(), nn * sizeof(R), cudaMemcpyHostToDevice);
                copy_(h_.touch[0] + o, tn.data(), nn, cudaMemcpyHostToDevice);
                copy_(h_.np[0] + o, pr.data(), nn * sizeof(int), cudaMemcpyHostToDevice);
                copy_(h_.rec[0] + 2 * o, rec.data(), 2 * nn * sizeof(int4), cudaMemcpyHostToDevice);
                copy_(S + 4 * o, sl.data(), 4 * nn * sizeof(R4<R>), cudaMemcpyHostToDevice);
            }
        }
        if (src && off != size) throw ArgError("checkpoint has trailing bytes");
    }
    void launch_info(int* step_loop, int* search_lanes, int* clump_batch, int* pair_blocks) override {
        if (step_loop) {
            if (opt_.use_graph && !loop_[0].tried) capture_loop(loop_[0]);
            *step_loop = loop_[0].exec ? 1 : 0;
        }
        if (search_lanes) *search_lanes = SEARCH_G;
        if (clump_batch) *clump_batch = 1;   // members per lane
        if (pair_blocks) *pair_blocks = pair_bps_;
    }
    void info(double* bytes, double* ms) override {
        if (bytes) *bytes = mem_.bytes;
        if (ms) *ms = last_ms_;
    }

   private:
    nbc_options opt_;
    bool shared_gpu_;        // a request server's, which steps several side by side (see step_grid)
    DevMem mem_;
    char* pslab_ = nullptr;  // the pair buffers' slab
    int3* relmap_ = nullptr; // [S] region moves of a re-layout
    size_t pslab_bytes_ = 0;
    char* xslab_ = nullptr;  // the export step's per-pair buffers (null until one runs)
    size_t xslab_bytes_ = 0;
    cudaStream_t stream_ = nullptr;
    cudaStream_t stream2_ = nullptr;   // second branch of a step: k_boundary beside k_pairs
    cudaEvent_t ev_fork_ = nullptr, ev_join_ = nullptr;
    Dev h_{};            // host copy of the device table
    Dev* d_ = nullptr;   // device table
    int S_ = 0, N_ = 0, K_ = 0;
    bool hgrid_ = false;
    bool sphere_any_ = false;   // some scene runs a sphere driver's behaviour (the clump pass's SPH build)
    bool sphere_kin_ = false;   // some scene runs the sphere drivers' kinematics (Dev::fint)
    bool has_kinds_ = false;    // some scene has split-driver body kinds (Dev::kind)
    bool first_list_ = true;
    int pair_bps_ = 12;      // blocks per SM of the pair kernel's grid
    int sm_count_ = 148;
    int ring_len_ = 1;
    std::vector<ScenePar> hpar_;
    std::vector<int> start_step_;
    // the engine's clump order (see clump_order): the caller's number within
    // its scene of each clump, the first member slot and the clump of each
    // member slot, and the member slot of each of the caller's subspheres
    std::vector<int> cold_, mstart_, mcl_, mrow_, clane_;   // clane_: first lane in Dev::lrec
    int* hflag_ = nullptr;  // pinned
    int steps_done_ = 0;
    int runs_before_ = 0;    // launches of k_steps before the ones enqueued
    int pend_ = 0, pend_eager_ = 0, pend_before_ = 0;  // steps enqueued and not yet waited for
    bool post_done_ = false;
    double last_ms_ = 0;
    // step graphs by timing level: [0] plain, [1] event nodes around the
    // contact pass (k_pairs + k_sum), [2] event nodes at every mark
    cudaGraph_t graph_[3] = {nullptr, nullptr, nullptr};
    cudaGraphExec_t gexec_[3] = {nullptr, nullptr, nullptr};
    // the untimed graph with a device-side step loop (capture_loop): [v] for an
    // engine that is one of up to 2^v stepping on the device (see step_grid),
    // made when needed
    struct Loop {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        cudaGraphNode_t init = nullptr;
        bool tried = false;
    };
    static constexpr int SHARES = 6;
    Loop loop_[SHARES];
    Loop* cur_ = &loop_[0];   // the one of the steps enqueued
    bool stepping_ = false;   // counted in g_stepping
    // the engine counts as stepping; which of its loops to take
    int enter_stepping() {
        std::atomic<int>& n = g_stepping[opt_.device & 63];
        const int all = stepping_ ? n.load() : n.fetch_add(1) + 1;
        stepping_ = true;
        int v = 0;
        while (!shared_gpu_ && v + 1 < SHARES && (1 << v) < all) v++;
        return v;
    }
    void leave_stepping() {
        if (stepping_) g_stepping[opt_.device & 63].fetch_sub(1);
        stepping_ = false;
    }
    // kernel timing: one record of NMARK events per step, at the marks
    //   0 step start  1 after k_clump  2 after the rebuild node
    //   3/4 around k_boundary and 5 start of the contact pass (second branch)
    //   6 end of the contact pass (after k_sum)  7 step end
    static constexpr int NMARK = 8;
    static constexpr int PH_CLUMP = 0, PH_REBUILD = 1, PH_BOUNDARY = 2, PH_CONTACT = 3, PH_STEP = 4, NPH = 5;
    int timing_ = 0;
    double t_phase_ms_[NPH] = {0, 0, 0, 0, 0};
    int t_contact_n_ = 0;
    long long launches_ = 0;
    int rebuilds_at_enable_ = 0;
    std::vector<cudaEvent_t> ev_;   // records of NMARK events
    int ev_used_ = 0;               // records made and not yet harvested
    cudaEvent_t* rec_ = nullptr;    // the record being made by an eager step (null: none)
    int capture_timed_ = 0;
    cudaEvent_t gev_[3][NMARK] = {};
    cudaGraphNode_t gev_node_[3][NMARK] = {};

    int total_rebuilds() {
        std::vector<SceneDyn> y(S_);
        copy_(y.data(), h_.dyn, S_ * sizeof(SceneDyn), cudaMemcpyDeviceToHost);
        int n = 0;
        for (auto& v : y) n = std::max(n, v.nrebuild);
        return n;
    }
    // kernels of one rebuild in a graph (launch_rebuild; the eager path adds a
    // k_need): plan, hash, the cell counts' scan, scatter, order, the two
    // searches, the rows' scan, fill, rows, commit
    int rebuild_launches() const { return S_ == 1 ? 9 : 11; }
    cudaEvent_t* next_record() {
        if ((size_t)(NMARK * (ev_used_ + 1)) > ev_.size()) {
            for (int k = 0; k < 64 * NMARK; k++) {
                cudaEvent_t e;
                CK(cudaEventCreate(&e));
                ev_.push_back(e);
            }
        }
        return &ev_[(size_t)NMARK * ev_used_++];
    }
    // marks recorded at timing level 1: only those around the contact pass
    static bool mark_on(int level, int k) { return level >= 2 || (level == 1 && (k == 5 || k == 6)); }
    void harvest_events() {
        for (int k = 0; k < ev_used_; k++) {
            const cudaEvent_t* e = &ev_[(size_t)NMARK * k];
            float ms[NPH] = {0, 0, 0, 0, 0};
            CK(cudaEventElapsedTime(&ms[PH_CONTACT], e[5], e[6]));
            if (timing_ >= 2) {
                CK(cudaEventElapsedTime(&ms[PH_CLUMP], e[0], e[1]));
                CK(cudaEventElapsedTime(&ms[PH_REBUILD], e[1], e[2]));
                CK(cudaEventElapsedTime(&ms[PH_BOUNDARY], e[3], e[4]));
                CK(cudaEventElapsedTime(&ms[PH_STEP], e[0], e[7]));
            }
            for (int p = 0; p < NPH; p++) t_phase_ms_[p] += ms[p];
            t_contact_n_++;
        }
        ev_used_ = 0;
    }
    // a timing mark on stream st: an event node while capturing a timed
    // graph, an event of the current record on an eager step
    void mark(int k, cudaStream_t st) {
        if (capturing_) {
            if (!mark_on(capture_timed_, k)) return;
            CK(cudaEventRecordWithFlags(gev_[capture_timed_][k], st, cudaEventRecordExternal));
            gev_node_[capture_timed_][k] = last_captured_node(st);
        } else if (rec_ && mark_on(timing_, k)) {
            CK(cudaEventRecord(rec_[k], st));
        }
    }

    struct RowData { std::vector<int> row, brow, nbr, bnbr, bpair; };

    // ---- setup --------------------------------------------------------------
    // The order in which the engine keeps a scene's clumps: by the grid cell
    // of the clump's first member (grid level, then z, y, x: the order of the
    // subspheres), ties in the caller's order.  Clumps that lie side by side
    // then share cache lines in the clump pass (its members' positions) and
    // in the pair kernel (velocities, lever arms).  It is kept for the
    // engine's life: a packed bed mixes slowly.  No result depends on it.
    static std::vector<int> clump_order(const nbc_scene_desc& D, const ScenePar& P) {
        std::vector<int> first(D.n_clump, -1);
        for (int i = D.n_sub - 1; i >= 0; i--) first[D.clump_id[i]] = i;
        std::vector<uint32_t> key(D.n_clump);
        for (int k = 0; k < D.n_clump; k++) {
            const int i = first[k];
            if (i < 0) { key[k] = 0xffffffffu; continue; }   // a clump without members
            const int lv = P.levels > 1 ? D.level[i] : 0;
            const int* dim = P.levels > 1 ? P.ldim[lv] : P.gdim;
            uint32_t c = 0;
            for (int a = 2; a >= 0; a--) {
                const double x = (D.pos[3 * i + a] - P.origin[a]) / (P.levels > 1 ? P.lcell[lv] : P.cell[a]);
                c = c * (uint32_t)dim[a] + (uint32_t)std::min(std::max(x, 0.0), (double)(dim[a] - 1));
            }
            key[k] = (P.levels > 1 ? (uint32_t)P.loff[lv] : 0u) + c;
        }
        // stable radix sort, 11 bits a pass
        std::vector<int> ord(D.n_clump), tmp(D.n_clump);
        for (int k = 0; k < D.n_clump; k++) ord[k] = k;
        for (int shift = 0; shift < 33; shift += 11) {
            int at[2049] = {0};
            for (int k = 0; k < D.n_clump; k++) at[((key[k] >> shift) & 2047) + 1]++;
            for (int b = 0; b < 2048; b++) at[b + 1] += at[b];
            for (int k : ord) tmp[at[(key[k] >> shift) & 2047]++] = k;
            ord.swap(tmp);
        }
        return ord;
    }
    void setup(const std::vector<const nbc_scene_desc*>& sc) {
        for (size_t s = 0; s < sc.size(); s++) validate_scene(*sc[s], (int)s);
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) throw CudaError("no CUDA device");
        CK(cudaSetDevice(opt_.device));
        CK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
        CK(cudaStreamCreateWithFlags(&stream2_, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&ev_fork_, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&ev_join_, cudaEventDisableTiming));
        hflag_ = g_pinned.get();
        mem_.stream = stream_;
        DevMem::keep_pool(opt_.device);
        pair_bps_ = opt_.pair_blocks >= 2 && opt_.pair_blocks <= 16 ? opt_.pair_blocks : 12;
        CK(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, opt_.device));
        S_ = (int)sc.size();
        hpar_.resize(S_);
        start_step_.resize(S_);
        std::vector<SceneDyn> hdyn(S_);
        int cells = 0;
        for (int s = 0; s < S_; s++) {
            const nbc_scene_desc& D = *sc[s];
            if (D.n_sub <= 0 || D.n_clump <= 0 || !D.pos || !D.radius || !D.clump_id)
                throw ArgError("scene " + std::to_string(s) + ": empty or missing arrays");
            ScenePar& P = hpar_[s];
            memset(&P, 0, sizeof(P));
            P.dt = D.dt; P.E = D.ymod; P.nu = D.prat; P.mu = D.frcoe; P.gravity = D.gravity;
            P.beta = D.beta; P.cohesion = D.cohesion; P.thresh = D.thresh;
            // LoadParameters (src/dem_subsphere_io.cu:143-145)
            const double lnCOR = std::log(D.normres), PI_REF = 3.14159265359;
            P.damping = 2.0 * std::sqrt(5.0 / 6.0) * lnCOR / std::sqrt(lnCOR * lnCOR + PI_REF * PI_REF);
            P.kn_fac = 2.0 * D.ymod / (3.0 * (1.0 - D.prat * D.prat));
            P.ks_fac = 2.0 * D.ymod / (1.0 + D.prat) / (2.0 - D.prat);
            P.bl = D.branch_len > 0 ? D.branch_len : 256;
            // SetMeshSize (src/dem_subsphere_io.cu:195-230)
            double rmax = 0;
            for (int i = 0; i < D.n_sub; i++) rmax = std::max(rmax, D.radius[i]);
            const double mesh = 3.0 * rmax;
            for (int a = 0; a < 3; a++) {
                P.cell[a] = mesh;
                P.icell[a] = 1.0 / mesh;
                P.origin[a] = D.world_origin[a] - mesh;
                double ws = D.world_size[a] + 2 * mesh;
                P.gdim[a] = (int)(unsigned)std::ceil(ws / mesh);
                P.box_lo[a] = D.box_lo[a];
                P.box_hi[a] = D.box_hi[a];
            }
            P.lrmax[0] = (float)rmax * 1.000001f;
            P.levels = D.levels > 1 ? D.levels : 1;
            if (P.levels > 1) hgrid_ = true;
            if (P.levels > MAX_LEVELS) throw ArgError("too many grid levels");
            if (P.levels == 1) {
                P.cellnum = P.gdim[0] * P.gdim[1] * P.gdim[2];
            } else {
                int off = 0;
                for (int l = 0; l < P.levels; l++) {
                    P.lcell[l] = D.level_cell[l];
                    P.licell[l] = 1.0 / P.lcell[l];
                    double rl = 0;
                    for (int i = 0; i < D.n_sub; i++)
                        if (D.level[i] == l) rl = std::max(rl, D.radius[i]);
                    P.lrmax[l] = (float)rl * 1.000001f;
                    for (int a = 0; a < 3; a++)
                        P.ldim[l][a] = (int)std::ceil((D.world_size[a] + 2 * mesh) / P.lcell[l]);
                    P.loff[l] = off;
                    off += P.ldim[l][0] * P.ldim[l][1] * P.ldim[l][2];
                }
                P.cellnum = off + 1;
                for (int l = 0; l < P.levels; l++)
                    for (int f = l + 1; f < P.levels; f++)
                        if (1.5 * ((double)P.lrmax[l] + P.lrmax[f]) >= P.lcell[l]) P.tight = 1;
            }
            P.inside = 1;
            for (int l = 0; l < P.levels; l++)
                for (int a = 0; a < 3; a++) {
                    const double ext = P.levels > 1 ? P.ldim[l][a] * P.lcell[l] : P.gdim[a] * P.cell[a];
                    if (!(P.box_lo[a] >= P.origin[a] && P.box_hi[a] - P.origin[a] <= ext * (1.0 - 1e-9))) P.inside = 0;
                }
            P.cell_off = cells;
            cells += P.cellnum;
            P.sub_off = N_;
            P.nsub = D.n_sub;
            P.clump_off = K_;
            P.nclump = D.n_clump;
            N_ += D.n_sub;
            K_ += D.n_clump;
            // walls
            P.wall = D.is_wall_force ? D.wall : WALL_NONE;
            if (P.wall == WALL_CUBE) {
                for (int a = 0; a < 3; a++) {
                    P.w_half[a] = D.cube_half[a]; P.w_c[a] = D.cube_centre[a];
                    P.w_v[a] = D.cube_vel[a]; P.w_w[a] = D.cube_angvel[a];
                }
            } else if (P.wall == WALL_CYL) {
                P.cyl_R = D.cyl_radius; P.cyl_H = D.cyl_half_height;
                for (int a = 0; a < 3; a++) {
                    P.cyl_axis[a] = D.cyl_axis[a]; P.w_c[a] = D.cyl_centre[a];
                    P.w_v[a] = D.cyl_vel[a]; P.w_w[a] = D.cyl_angvel[a];
                }
            }
            SceneDyn& Y = hdyn[s];
            memset(&Y, 0, sizeof(Y));
            Y.rebuild = 1;  // the first step always builds the list (src/dem_simulation_clump.cu:124)
            P.has_intr = D.intruder == NBC_INTR_SPHERE || D.intruder == NBC_INTR_CYLINDER;
            if (P.has_intr) {
                P.intr_shape = D.intruder;
                P.intr_motion = D.intr_motion == NBC_MOTION_CONSTANT_VELOCITY ? 0 : 1;
                P.intr_wait = D.intr_motion == NBC_MOTION_GRAVITY_AFTER_CONTACT;
                P.intr_R = D.intr_radius;
                P.intr_H = D.intruder == NBC_INTR_SPHERE ? D.intr_radius : D.intr_half_height;
                for (int a = 0; a < 3; a++) {
                    P.intr_axis[a] = D.intr_axis[a];
                    P.intr_w[a] = D.intr_angvel[a];
                    Y.intr_p[a] = D.intr_pos[a];
                    Y.intr_v[a] = D.intr_vel[a];
                }
                P.intr_mass = D.intr_prop[3];
            }
            // the reference's sphere-only drivers (class DEMmain)
            if (D.sphere_mode & ~(NBC_SPHERE_KINEMATICS | NBC_SPHERE_CUBE_WALL | NBC_SPHERE_RESET_HISTORY))
                throw ArgError("scene " + std::to_string(s) + ": unknown sphere_mode bits");
            P.sphere = D.sphere_mode | (D.body_kind ? SPH_KINDS : 0);
            if (P.sphere) {
                // one-sphere clumps with the member at the centre: the clump
                // kinematics are then the sphere kinematics
                if (D.n_sub != D.n_clump)
                    throw ArgError("scene " + std::to_string(s) + ": sphere drivers need one subsphere per clump");
                std::vector<char> seen(D.n_clump, 0);
                for (int i = 0; i < D.n_sub; i++) {
                    const int c = D.clump_id[i];
                    if (c < 0 || c >= D.n_clump || seen[c] || D.local[3 * i] != 0.0 || D.local[3 * i + 1] != 0.0 ||
                        D.local[3 * i + 2] != 0.0)
                        throw ArgError("scene " + std::to_string(s) +
                                       ": sphere drivers need one subsphere per clump at its centre (LocalPos = 0)");
                    seen[c] = 1;
                }
            }
            if (P.sphere) sphere_any_ = true;
            if (P.sphere & SPH_KIN) sphere_kin_ = true;
            if (P.sphere & SPH_KINDS) {
                for (int k = 0; k < D.n_clump; k++)
                    if (D.body_kind[k] < 0 || D.body_kind[k] > 2)
                        throw ArgError("scene " + std::to_string(s) + ": body kind out of range at clump " +
                                       std::to_string(k));
                has_kinds_ = true;
                // bodies of kind 1 move without triggering a rebuild: every
                // listed pair stays in the contact pass (near margin unbounded)
                P.thresh = 1e100;
            }
            start_step_[s] = D.start_step;
            ring_len_ = std::max(ring_len_, std::max(1, D.output_interval));
        }
        ring_len_ = std::max(ring_len_, 1024);
        // list entries keep two flag bits above the subsphere index
        if ((long long)N_ >= (1LL << 30)) throw ArgError("more than 2^30 subspheres in one engine");
        h_.S = S_; h_.N = N_; h_.K = K_;
        h_.cells = cells;
        h_.turn = step_turn();

        // host arrays: subspheres in the input order, clumps in the engine's
        std::vector<int> fix(N_), lev(N_, 0), sid(N_), csid(K_);
        std::vector<int2> cm(N_);
        std::vector<int> kind(has_kinds_ ? K_ : 0, 0);
        cold_.resize(K_);
        mstart_.assign(K_ + 1, 0);
        mcl_.resize(N_);
        mrow_.resize(N_);
        for (int s = 0; s < S_; s++) {
            const nbc_scene_desc& D = *sc[s];
            const ScenePar& P = hpar_[s];
            const std::vector<int> old = clump_order(D, P);
            std::vector<int> now(D.n_clump);
            for (int c = 0; c < D.n_clump; c++) {
                const int g = P.clump_off + c, k = old[c];
                now[k] = g;
                cold_[g] = k;
                csid[g] = s;
                // bits 0-1: Type; bits 2-3: the kind the split driver's first
                // half-kick sees, the body's original index (0, 1, 2, or 3 for
                // any larger index; see k_clump)
                if (has_kinds_ && D.body_kind) kind[g] = D.body_kind[k] | (std::min(k, 3) << 2);
            }
            for (int i = 0; i < D.n_sub; i++) {
                int g = P.sub_off + i;
                cm[g].x = now[D.clump_id[i]];
                fix[g] = i;
                sid[g] = s;
                if (P.levels > 1) lev[g] = D.level[i];
                mstart_[cm[g].x + 1]++;
            }
        }
        for (int k = 0; k < K_; k++) mstart_[k + 1] += mstart_[k];
        {
            std::vector<int> cur(mstart_.begin(), mstart_.end() - 1);
            for (int s = 0; s < S_; s++) {
                const nbc_scene_desc& D = *sc[s];
                for (int i = 0; i < D.n_sub; i++) {
                    const int g = hpar_[s].sub_off + i, k = cm[g].x, m = cur[k]++;
                    cm[g].y = m;
                    mcl_[m] = k;
                    mrow_[g] = m;
                }
            }
        }

        // the clump pass's lanes: whole clumps packed into warps, a lane per
        // member (a clump of more than 32 has a warp of its own, one without
        // members a lane)
        clane_.resize(K_);
        size_t lanes = 0;
        for (int k = 0; k < K_; k++) {
            const int nm = mstart_[k + 1] - mstart_[k], n = std::min(std::max(nm, 1), 32);
            if (lanes % 32 + n > 32) lanes = (lanes + 31) / 32 * 32;
            clane_[k] = (int)lanes;
            lanes += n;
            if (nm > 32) lanes = (lanes + 31) / 32 * 32;
        }
        h_.W = cdiv(lanes, 32);

        // device allocation: the per-subsphere and per-clump buffers in one
        // slab, the pair buffers (which grow) in another
        const size_t N = N_;
        auto layout = [&](Carver& m) {
            h_.par = m.take<ScenePar>(S_);
            h_.dyn = m.take<SceneDyn>(S_);
            h_.sid = m.take<int>(N);
            h_.csid = m.take<int>(K_);
            h_.posr = m.take<double4>(N); h_.posr2 = m.take<double4>(N);
            h_.cm = m.take<int2>(N); h_.cm2 = m.take<int2>(N);
            h_.part_fix = m.take<int>(N); h_.part_fix2 = m.take<int>(N);
            h_.level = m.take<int>(N); h_.level2 = m.take<int>(N);
            h_.key = m.take<int>(N); h_.key2 = m.take<int>(N);
            h_.lom = m.take<double4>(N); h_.cum = m.take<double4>(N); h_.kin = m.take<double4>(N);
            h_.bhist = m.take<R4<R>>((size_t)NB_SLOTS * 3 * N); h_.bhist2 = m.take<R4<R>>((size_t)NB_SLOTS * 3 * N);
            h_.bbits = m.take<uint16_t>(N); h_.bbits2 = m.take<uint16_t>(N);
            h_.fsum = m.take<R4<R>>(2 * N);
            h_.fbnd = m.take<R4<R>>(2 * N);
            h_.fint = sphere_kin_ ? m.take<R4<R>>(2 * N) : nullptr;
            h_.kind = has_kinds_ ? m.take<int>(K_) : nullptr;
            h_.cpos = m.take<double4>(K_); h_.cvel = m.take<double4>(K_); h_.cw = m.take<double4>(K_);
            h_.cq = m.take<double4>(K_); h_.cprop = m.take<double4>(K_);
            h_.cinv = m.take<double4>(K_);
            h_.lrec = m.take<int4>(2 * 32 * (size_t)h_.W); h_.clane = m.take<int>(K_);
            h_.cold = m.take<int>(K_); h_.stage = m.take<double4>(5 * (size_t)K_);
            h_.cF = m.take<double4>(K_); h_.cT = m.take<double4>(K_);
            h_.mem_start = m.take<int>(K_ + 1);
            h_.mo = m.take<int2>(N);
            int* flags = m.take<int>(FL_SIZE);
            h_.post_pending = flags + FL_POST;
            h_.any_rebuild = flags + FL_REBUILD;
            h_.halt = flags + FL_HALT;
            h_.step_base = flags + FL_BASE;
            h_.hgen = flags + FL_HGEN;
            h_.gstep = flags + FL_GSTEP;
            h_.kc_done = flags + FL_KC_DONE;
            h_.lstep = flags + FL_LSTEP;
            h_.loop_left = flags + FL_LEFT;
            h_.scan_fail = flags + FL_SCAN_FAIL;
            h_.step_phase = flags + FL_PHASE;
            h_.step_runs = flags + FL_STEP_RUNS;
            h_.step_bar = (unsigned long long*)(flags + FL_BAR);
            h_.kA = m.take<int>(N); h_.vA = m.take<int>(N); h_.vB = m.take<int>(N);
            h_.posf = m.take<float4>(N);
            h_.ccnt = m.take<int>((size_t)cells + S_ + 1);
            h_.perm = m.take<int>(N);
            h_.inv = m.take<int>(N);
            h_.cstart = m.take<int>(cells + 1);
            h_.scr = m.take<int>((size_t)N * SCR_CAP);
            h_.rlong = m.take<uint8_t>(N);
            h_.cnt_f = m.take<int>(N + 1); h_.cnt_b = m.take<int>(N + 1); h_.cnt_nf = m.take<int>(N + 1);
            h_.cnt_ns = m.take<int>(N + 1); h_.xcnt = m.take<int>(N + 1);
            h_.fcur = m.take<int>(N);
            h_.nsl = m.take<int2>(N);
            h_.nprefix = m.take<int>(S_ + 1);
            h_.bidx = m.take<int>(N);
            h_.bprefix = m.take<int>(S_ + 1);
            const long long scan_tiles = std::max(cdiv(N + 1, SC_TILE), cdiv((long long)cells + S_ + 1, SC_TILE));
            h_.scan_st = m.take<unsigned long long>(5 * scan_tiles + 5);
            h_.scan_ctl = m.take<int>(2);
            for (int l = 0; l < 2; l++) {
                h_.L[l].row = m.take<int>(N + S_);
                h_.L[l].brow = m.take<int>(N + S_);
                h_.nro[l] = m.take<int>(N + S_);
            }
            h_.plan = m.take<int>(PL_SIZE);
            h_.pscene = m.take<int>(S_);
            h_.psub = m.take<int>(S_ + 1);
            h_.pcell = m.take<int>(S_ + 1);
            h_.pwarp = m.take<int>(S_ + 1);
            h_.need = m.take<int>(S_);
            relmap_ = m.take<int3>(S_);
            h_.xparts = m.take<R4<R>>(6 * N);
            h_.xintr = m.take<R4<R>>(4 * N);
            h_.ring_len = ring_len_;
            h_.ring = m.take<double>((size_t)S_ * ring_len_ * 6);
            d_ = m.take<Dev>(1);
        };
        Carver sz;
        layout(sz);
        Carver m{(uintptr_t)mem_.alloc<char>(sz.off)};
        layout(m);
        // the pair regions are sized at the first list (nothing is stored in them before)
        alloc_pairs(1);

        copy_(h_.par, hpar_.data(), S_ * sizeof(ScenePar), cudaMemcpyHostToDevice);
        copy_(h_.dyn, hdyn.data(), S_ * sizeof(SceneDyn), cudaMemcpyHostToDevice);
        if (S_ > 1) {   // (the slab is zeroed)
            copy_(h_.sid, sid.data(), N * sizeof(int), cudaMemcpyHostToDevice);
            copy_(h_.csid, csid.data(), K_ * sizeof(int), cudaMemcpyHostToDevice);
        }
        copy_(h_.cm, cm.data(), N * sizeof(int2), cudaMemcpyHostToDevice);
        copy_(h_.part_fix, fix.data(), N * sizeof(int), cudaMemcpyHostToDevice);
        if (hgrid_) copy_(h_.level, lev.data(), N * sizeof(int), cudaMemcpyHostToDevice);
        // the caller's arrays go up as they are (several scenes': one after the
        // other) and are packed into records and put in place on the device
        std::vector<double> joined;
        auto upload = [&](double* dst, const double* nbc_scene_desc::*field, bool members, int width) {
            const size_t total = (size_t)width * (members ? N_ : K_);
            const double* src = sc[0]->*field;
            if (S_ > 1) {
                joined.resize(total);
                for (int s = 0; s < S_; s++) {
                    const ScenePar& P = hpar_[s];
                    memcpy(&joined[(size_t)width * (members ? P.sub_off : P.clump_off)], sc[s]->*field,
                           sizeof(double) * width * (members ? P.nsub : P.nclump));
                }
                src = joined.data();
            }
            copy_(dst, src, total * sizeof(double), cudaMemcpyHostToDevice);
        };
        double *so = (double*)h_.posr2, *sp = (double*)h_.kin;   // 4 N doubles each, not in use yet
        upload(so, &nbc_scene_desc::local, true, 3);
        upload(so + 3 * N, &nbc_scene_desc::mass, true, 1);
        upload(sp, &nbc_scene_desc::pos, true, 3);
        upload(sp + 3 * N, &nbc_scene_desc::radius, true, 1);
        k_members_up<<<std::min(cdiv(N_, 256), sm_count_ * 8), 256, 0, stream_>>>(so, sp, h_.cm, N_, h_.lom, h_.posr);
        CK(cudaGetLastError());
        CK(cudaMemsetAsync(h_.kin, 0, N * sizeof(double4), stream_));
        {
            std::vector<int> abs(K_);
            for (int s = 0; s < S_; s++)
                for (int c = hpar_[s].clump_off; c < hpar_[s].clump_off + hpar_[s].nclump; c++)
                    abs[c] = hpar_[s].clump_off + cold_[c];
            copy_(h_.cold, abs.data(), K_ * sizeof(int), cudaMemcpyHostToDevice);
        }
        double* st = (double*)h_.stage;
        upload(st, &nbc_scene_desc::clump_pos, false, 3);
        upload(st + 3 * (size_t)K_, &nbc_scene_desc::clump_vel, false, 3);
        upload(st + 6 * (size_t)K_, &nbc_scene_desc::clump_angvel, false, 3);
        upload(st + 9 * (size_t)K_, &nbc_scene_desc::clump_quat, false, 4);
        upload(st + 13 * (size_t)K_, &nbc_scene_desc::clump_prop, false, 4);
        if (h_.kind) copy_(h_.kind, kind.data(), K_ * sizeof(int), cudaMemcpyHostToDevice);
        copy_(h_.clane, clane_.data(), K_ * sizeof(int), cudaMemcpyHostToDevice);
        copy_(h_.mem_start, mstart_.data(), (K_ + 1) * sizeof(int), cudaMemcpyHostToDevice);
        // the first list is empty: rows of zeros (the slab is zeroed)
        int one = 1;
        copy_(h_.any_rebuild, &one, sizeof(int), cudaMemcpyHostToDevice);
        push_dev();
        const int g = std::min(cdiv(std::max(N_, 32 * h_.W), 256), sm_count_ * 8);
        k_clumps_up<<<std::min(cdiv(K_, 256), sm_count_ * 8), 256, 0, stream_>>>(d_);
        k_members_init<<<g, 256, 0, stream_>>>(d_);
        k_lanes_init<<<g, 256, 0, stream_>>>(d_);
        CK(cudaGetLastError());
    }

    void alloc_pairs(long long cap) {
        if (cap > 2000000000LL) throw CudaError("pair capacity above 2^31");
        h_.cap = (int)cap;
        auto layout = [&](Carver& m) {
            for (int l = 0; l < 2; l++) {
                h_.L[l].nbr = m.take<int>(cap);
                h_.L[l].own = m.take<int>(cap);
                h_.L[l].bnbr = m.take<int>(cap);
                h_.L[l].bpair = m.take<int>(cap);
                h_.H[l] = m.take<char>(hist_bytes(cap));
                h_.touch[l] = m.take<uint8_t>(cap);
                h_.rec[l] = m.take<int4>(2 * cap);
                h_.np[l] = m.take<int>(cap);
            }
            h_.slots = m.take<R4<R>>(4 * cap);
            h_.tmp = m.take<int2>(cap);
            h_.bslot = m.take<int>(cap);
        };
        // the export step's pair buffers are made when one runs
        if (xslab_) mem_.release(xslab_, xslab_bytes_);
        xslab_ = nullptr;
        h_.xfcn = h_.xcpt = nullptr;
        Carver sz;
        layout(sz);
        pslab_bytes_ = sz.off;
        pslab_ = mem_.alloc<char>(pslab_bytes_);
        Carver m{(uintptr_t)pslab_};
        layout(m);
    }
    void alloc_export() {
        if (xslab_) return;
        refresh_dev();
        auto layout = [&](Carver& m) {
            h_.xfcn = m.take<R4<R>>(h_.cap);
            h_.xcpt = m.take<double4>(h_.cap);
        };
        Carver sz;
        layout(sz);
        xslab_bytes_ = sz.off;
        xslab_ = mem_.alloc<char>(xslab_bytes_);
        Carver m{(uintptr_t)xslab_};
        layout(m);
        push_dev();
    }
    static size_t hist_bytes(long long cap) { return (size_t)cap * (2 * sizeof(R4<R>) + sizeof(R)); }

    double slack() const { return opt_.pair_slack >= 1.0 ? opt_.pair_slack : 1.6; }
    // Bytes of the pair buffers per pair slot.
    static double bytes_per_pair() {
        return 2.0 * (5 * sizeof(int) + (double)hist_bytes(1) + 1 + 2 * sizeof(int4)) + 4 * sizeof(R4<R>) +
               sizeof(int2) + sizeof(int);
    }
    // Region capacities for the first lists: slack x each scene's pairs; with
    // the default slack at least the reference's own list capacity, n_sub x
    // BranchLmtLen/2, as far as 30% of the free device memory allows (growing
    // later costs a host round trip and a re-layout).
    std::vector<long long> first_capacities(const std::vector<long long>& need) {
        std::vector<long long> cap(S_);
        for (int s = 0; s < S_; s++) cap[s] = std::max<long long>(16, (long long)std::ceil(need[s] * slack()));
        if (opt_.pair_slack >= 1.0) return cap;
        double want = 0, have = 0;
        for (int s = 0; s < S_; s++) {
            have += (double)cap[s];
            want += std::max(0.0, (double)hpar_[s].nsub * (hpar_[s].bl / 2) - (double)cap[s]);
        }
        size_t fr = 0, tot = 0;
        CK(cudaMemGetInfo(&fr, &tot));
        const double budget = 0.3 * (double)fr / bytes_per_pair() - have;
        if (budget <= 0 || want <= 0) return cap;
        const double f = std::min(1.0, budget / want);
        for (int s = 0; s < S_; s++) {
            const double extra = std::max(0.0, (double)hpar_[s].nsub * (hpar_[s].bl / 2) - (double)cap[s]);
            cap[s] += (long long)(f * extra);
        }
        return cap;
    }
    // the regions after an overflow: every scene whose new list does not fit
    // gets slack x its pairs (at least 1,024 more slots)
    std::vector<long long> grown_capacities(const std::vector<int>& need, const std::vector<SceneDyn>& y) {
        std::vector<long long> cap(S_);
        for (int s = 0; s < S_; s++) {
            cap[s] = y[s].pcap;
            if (need[s] > y[s].pcap)
                cap[s] = std::max<long long>((long long)std::ceil(need[s] * slack()), (long long)y[s].pcap + 1024);
        }
        return cap;
    }
    std::vector<SceneDyn> read_dyn_all() {
        std::vector<SceneDyn> y(S_);
        copy_(y.data(), h_.dyn, S_ * sizeof(SceneDyn), cudaMemcpyDeviceToHost);
        return y;
    }
    // New pair regions of the given capacities: the pair buffers are
    // re-allocated and every scene's current list, work records, histories
    // and touch flags move to its new region (rows shifted).  The build
    // buffers need nothing: a rebuild writes them before reading.
    void layout_pairs(const std::vector<long long>& pcap) {
        refresh_dev();
        std::vector<SceneDyn> y = read_dyn_all();
        std::vector<int3> map(S_);
        long long total = 0;
        int moved = 0;
        for (int s = 0; s < S_; s++) {
            map[s].x = y[s].pair_off;
            map[s].y = (int)total;
            map[s].z = moved;
            moved += y[s].npairs;
            y[s].pair_off = (int)total;
            y[s].pcap = (int)pcap[s];
            total += pcap[s];
            if (total > 2000000000LL) throw CudaError("pair capacity above 2^31");
        }
        Dev old = h_;
        char* old_slab = pslab_;
        const size_t old_bytes = pslab_bytes_;
        alloc_pairs(std::max<long long>(total, 1));
        copy_(h_.dyn, y.data(), S_ * sizeof(SceneDyn), cudaMemcpyHostToDevice);
        copy_(relmap_, map.data(), S_ * sizeof(int3), cudaMemcpyHostToDevice);
        push_dev();
        const int B = 256;
        if (moved > 0)
            k_relayout<R><<<std::min(148 * 8, cdiv(moved, B)), B, 0, stream_>>>(d_, old, relmap_, moved);
        k_shift_rows<<<std::min(148 * 8, cdiv((long long)N_ + S_, B)), B, 0, stream_>>>(d_, relmap_);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(stream_));
        mem_.release(old_slab, old_bytes);
    }

    // Every copy goes through the engine's own stream.  cudaMemcpy would run
    // on the legacy default stream, which is not ordered with the engine's
    // non-blocking streams: a device-to-device copy (and the DMA of a pageable
    // host-to-device copy) may still be in flight when cudaMemcpy returns, so
    // a later kernel, or a stream-ordered free of the source, would race it.
    // Copies that touch host memory wait for the stream before returning.
    void copy_(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
        if (!bytes) return;
        CK(cudaMemcpyAsync(dst, src, bytes, kind, stream_));
        if (kind != cudaMemcpyDeviceToDevice) CK(cudaStreamSynchronize(stream_));
    }
    void push_dev() {
        CK(cudaStreamSynchronize(stream_));
        copy_(d_, &h_, sizeof(Dev), cudaMemcpyHostToDevice);
    }
    // the host copy of the pointer table, as the device has it
    void refresh_dev() {
        CK(cudaStreamSynchronize(stream_));
        copy_(&h_, d_, sizeof(Dev), cudaMemcpyDeviceToHost);
    }
    int read_int(const int* p) {
        CK(cudaStreamSynchronize(stream_));
        int v = 0;
        copy_(&v, p, sizeof(int), cudaMemcpyDeviceToHost);
        return v;
    }
    // the device's words for the steps, one after the other, in one copy (a
    // blocking copy is 10 us: five of them were a third of a call of one step)
    enum { FL_POST, FL_REBUILD, FL_HALT, FL_BASE, FL_HGEN, FL_GSTEP, FL_KC_DONE, FL_LSTEP, FL_LEFT, FL_SCAN_FAIL,
           FL_PHASE, FL_STEP_RUNS, FL_BAR, FL_SIZE = FL_BAR + 2 };
    struct Flags {
        int v[FL_SIZE];
    };
    Flags read_flags() {
        Flags f;
        copy_(&f, h_.post_pending, sizeof(f), cudaMemcpyDeviceToHost);
        return f;
    }
    SceneDyn read_dyn(int s) {
        CK(cudaStreamSynchronize(stream_));
        SceneDyn y;
        copy_(&y, h_.dyn + s, sizeof(SceneDyn), cudaMemcpyDeviceToHost);
        return y;
    }
    void pull_r4(const void* base, int off, int n, double* dst) {
        if (!dst) return;
        std::vector<R4<R>> tmp(n);
        copy_(tmp.data(), (const R4<R>*)base + off, n * sizeof(R4<R>), cudaMemcpyDeviceToHost);
        for (int i = 0; i < n; i++) { dst[3 * i] = tmp[i].x; dst[3 * i + 1] = tmp[i].y; dst[3 * i + 2] = tmp[i].z; }
    }
    RowData pull_rows(int s) {
        refresh_dev();
        const ScenePar& P = hpar_[s];
        const PairList& Lc = h_.L[0];
        RowData rd;
        rd.row.resize(P.nsub + 1);
        rd.brow.resize(P.nsub + 1);
        copy_(rd.row.data(), Lc.row + P.sub_off + s, (P.nsub + 1) * sizeof(int), cudaMemcpyDeviceToHost);
        copy_(rd.brow.data(), Lc.brow + P.sub_off + s, (P.nsub + 1) * sizeof(int), cudaMemcpyDeviceToHost);
        int nf = rd.row[P.nsub] - rd.row[0], nb = rd.brow[P.nsub] - rd.brow[0];
        rd.nbr.resize(nf);
        rd.bnbr.resize(nb);
        rd.bpair.resize(nb);
        copy_(rd.nbr.data(), Lc.nbr + rd.row[0], nf * sizeof(int), cudaMemcpyDeviceToHost);
        copy_(rd.bnbr.data(), Lc.bnbr + rd.brow[0], nb * sizeof(int), cudaMemcpyDeviceToHost);
        copy_(rd.bpair.data(), Lc.bpair + rd.brow[0], nb * sizeof(int), cudaMemcpyDeviceToHost);
        return rd;
    }

    // (w: Dev::scan_fail)
    static void check_wait(int w) {
        if (w == WAIT_BARRIER) throw CudaError("the step loop gave up waiting at its grid barrier (step halted)");
        if (w) throw CudaError("a list-rebuild scan gave up waiting on a tile (step halted)");
    }
    void check_errors() {
        std::vector<SceneDyn> y(S_);
        copy_(y.data(), h_.dyn, S_ * sizeof(SceneDyn), cudaMemcpyDeviceToHost);
        for (int s = 0; s < S_; s++)
            if (y[s].err & ERR_NONFINITE) throw NonFinite("scene " + std::to_string(s) + ": non-finite force");
    }

    // ---- launches -------------------------------------------------------------
    void launch_clump(int do_pre, cudaGraphConditionalHandle cond = 0, int use_cond = 0) {
        const int g = cdiv(h_.W + cdiv(S_, 32), CL_WARPS);
        if (sphere_any_) k_clump<R, true><<<g, CL_THREADS, 0, stream_>>>(d_, do_pre, cond, use_cond);
        else k_clump<R, false><<<g, CL_THREADS, 0, stream_>>>(d_, do_pre, cond, use_cond);
        CK(cudaGetLastError());
        if (!capturing_) launches_ += 1;
    }
    bool capturing_ = false;
    // the contact pass: k_pairs, with k_boundary beside it on the second
    // stream (fork and join by events, which become graph edges when
    // captured), then k_sum
    void launch_contact(bool exp) {
        if (exp) {
            alloc_export();
            CK(cudaMemsetAsync(h_.xfcn, 0, (size_t)h_.cap * sizeof(R4<R>), stream_));
            CK(cudaMemsetAsync(h_.xcpt, 0, (size_t)h_.cap * sizeof(double4), stream_));
            // wall and intruder parts: k_boundary writes its candidates only
            CK(cudaMemsetAsync((R4<R>*)h_.xparts + 2 * (size_t)N_, 0, 4 * (size_t)N_ * sizeof(R4<R>), stream_));
            CK(cudaMemsetAsync(h_.xintr, 0, 4 * (size_t)N_ * sizeof(R4<R>), stream_));
        }
        CK(cudaEventRecord(ev_fork_, stream_));
        CK(cudaStreamWaitEvent(stream2_, ev_fork_, 0));
        // the start of the contact pass is marked on the side branch (same
        // dependencies), so only its end mark sits on the critical path
        mark(5, stream2_);
        mark(3, stream2_);
        // grid-stride over the boundary candidates (a device count)
        const int bg = std::min(sm_count_ * 8, cdiv(N_, BD_THREADS));
        if (sphere_any_) {
            if (exp) k_boundary<R, true, true><<<bg, BD_THREADS, 0, stream2_>>>(d_);
            else k_boundary<R, false, true><<<bg, BD_THREADS, 0, stream2_>>>(d_);
        } else if (exp) k_boundary<R, true, false><<<bg, BD_THREADS, 0, stream2_>>>(d_);
        else k_boundary<R, false, false><<<bg, BD_THREADS, 0, stream2_>>>(d_);
        mark(4, stream2_);
        CK(cudaEventRecord(ev_join_, stream2_));
        // grid-stride over the near pairs (a device count), so a fixed grid
        // stays valid as the list grows; a small scene gets a small grid so
        // that other scenes' kernels run beside it
        const int pg = std::min(sm_count_ * pair_bps_, cdiv(3LL * N_, PR_THREADS));
        if (exp) k_pairs<R, true><<<pg, PR_THREADS, 0, stream_>>>(d_);
        else k_pairs<R, false><<<pg, PR_THREADS, 0, stream_>>>(d_);
        CK(cudaStreamWaitEvent(stream_, ev_join_, 0));
        CK(cudaGetLastError());
        mark(6, stream_);
        if (!capturing_) launches_ += CONTACT_LAUNCHES;
        // the export step also records the per-subsphere pair part
        if (exp) launch_sum(true);
    }
    // per-subsphere totals of the last contact pass into fsum (the clump
    // pass sums the same slots itself; this runs for getters and exports)
    void launch_sum(bool exp) {
        if (exp) k_sum<R, true><<<cdiv(N_, CT_THREADS), CT_THREADS, 0, stream_>>>(d_);
        else k_sum<R, false><<<cdiv(N_, CT_THREADS), CT_THREADS, 0, stream_>>>(d_);
        CK(cudaGetLastError());
    }
    // exclusive scans of arrays of the same length over [0, n), or over
    // [0, *dn) when dn is given (n then bounds it), in one launch
    void scan(std::initializer_list<int*> arrays, int n, const int* dn = nullptr) {
        ScanArrays a{};
        for (int* p : arrays) a.a[a.n++] = p;
        // a grid of at most a few blocks per SM takes the tiles; a grid sized
        // for the largest length would start tens of thousands of blocks that
        // find nothing to do when few scenes are rebuilt
        const int nb = std::min(std::max(1, cdiv(n, SC_TILE)) * a.n, sm_count_ * 4);
        k_scan1<<<nb, SC_THREADS, 0, stream_>>>(a, n, dn, h_.scan_st, h_.scan_ctl, h_.halt, h_.scan_fail);
    }
    // The rebuild block of src/dem_simulation_clump.cu:124-176, over the
    // scenes whose rebuild flag is set: every kernel but the near rows walks
    // the rebuilt scenes only (grid-stride over counts the plan puts on the
    // device), so a batch pays for the scenes it rebuilds.
    void launch_rebuild(bool eager) {
        const int B = 128;
        const int gN = std::min(cdiv(N_ + 1, B), sm_count_ * 16);         // grid-stride grids
        const int* pl = h_.plan;
        if (S_ > 1) k_plan<<<1, SC_THREADS, 0, stream_>>>(d_);
        k_hash<<<gN, B, 0, stream_>>>(d_);
        scan({h_.ccnt}, h_.cells + S_ + 1, pl + PL_TC1);
        k_cscatter<<<gN, B, 0, stream_>>>(d_);
        k_order<R><<<gN, B, 0, stream_>>>(d_);
        const int gS = std::min(cdiv((long long)N_ * SEARCH_G, SEARCH_THREADS), sm_count_ * 16);
        k_search<<<gS, SEARCH_THREADS, 0, stream_>>>(d_);
        k_search_faces<<<std::min(gS, sm_count_ * 4), SEARCH_THREADS, 0, stream_>>>(d_);
        scan({h_.cnt_f, h_.cnt_b, h_.cnt_nf, h_.cnt_ns, h_.xcnt}, N_ + 1, pl + PL_T1);
        CK(cudaGetLastError());
        if (eager) {
            // size the regions to the first lists, or grow the ones that overflow
            k_need<<<1, 256, 0, stream_>>>(d_);
            CK(cudaStreamSynchronize(stream_));
            check_wait(read_int(h_.scan_fail));
            std::vector<int> need(S_);
            copy_(need.data(), h_.need, S_ * sizeof(int), cudaMemcpyDeviceToHost);
            std::vector<SceneDyn> y = read_dyn_all();
            if (first_list_) {
                std::vector<long long> nd(S_);
                for (int s = 0; s < S_; s++) nd[s] = need[s] >= 0 ? need[s] : y[s].npairs;
                layout_pairs(first_capacities(nd));
                first_list_ = false;
            } else {
                bool grow = false;
                for (int s = 0; s < S_; s++) grow |= need[s] > y[s].pcap;
                if (grow) layout_pairs(grown_capacities(need, y));
            }
        }
        k_fill<<<gS, SEARCH_THREADS, 0, stream_>>>(d_);
        k_rows<R><<<std::min(cdiv(8LL * N_, SEARCH_THREADS), sm_count_ * 16), SEARCH_THREADS, 0, stream_>>>(d_, d_);
        if (S_ > 1)
            k_commit<R><<<std::min(sm_count_ * 4, cdiv(8LL * N_, SC_THREADS)), SC_THREADS, 0, stream_>>>(d_);
        CK(cudaGetLastError());
    }

    void run_step_eager(bool exp) {
        rec_ = timing_ ? next_record() : nullptr;
        mark(0, stream_);
        launch_clump(1);
        mark(1, stream_);
        CK(cudaMemcpyAsync(hflag_, h_.any_rebuild, sizeof(int), cudaMemcpyDeviceToHost, stream_));
        CK(cudaStreamSynchronize(stream_));
        if (hflag_[0]) launch_rebuild(true);
        mark(2, stream_);
        launch_contact(exp);
        mark(7, stream_);
        rec_ = nullptr;
        steps_done_ += 1;
    }

    // one step as a graph: k_clump, a conditional node holding the rebuild,
    // then k_boundary and k_contact on two branches; the timed variants have
    // event nodes at the timing marks
    void capture(int timed) {
        if (timed && !gev_[timed][0])
            for (int k = 0; k < NMARK; k++) CK(cudaEventCreate(&gev_[timed][k]));
        capturing_ = true;
        capture_timed_ = timed;
        cudaGraph_t& graph = graph_[timed];
        CK(cudaGraphCreate(&graph, 0));
        cudaGraphConditionalHandle hnd;
        CK(cudaGraphConditionalHandleCreate(&hnd, graph, 0, cudaGraphCondAssignDefault));
        CK(cudaStreamBeginCaptureToGraph(stream_, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        mark(0, stream_);
        launch_clump(1, hnd, 1);
        mark(1, stream_);
        cudaStreamCaptureStatus st;
        const cudaGraphNode_t* deps = nullptr;
        size_t ndeps = 0;
        CK(cudaStreamGetCaptureInfo(stream_, &st, nullptr, nullptr, &deps, &ndeps));
        cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
        cp.conditional.handle = hnd;
        cp.conditional.type = cudaGraphCondTypeIf;
        cp.conditional.size = 1;
        cudaGraphNode_t cnode;
        CK(cudaGraphAddNode(&cnode, graph, deps, ndeps, &cp));
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        CK(cudaStreamUpdateCaptureDependencies(stream_, &cnode, 1, cudaStreamSetCaptureDependencies));
        mark(2, stream_);
        launch_contact(false);
        mark(7, stream_);
        cudaGraph_t g2 = nullptr;
        CK(cudaStreamEndCapture(stream_, &g2));
        // the rebuild branch
        capture_timed_ = 0;
        CK(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        launch_rebuild(false);
        cudaGraph_t b2 = nullptr;
        CK(cudaStreamEndCapture(stream_, &b2));
        capturing_ = false;
        for (int k = 0; k < NMARK; k++)
            if (mark_on(timed, k) && !gev_node_[timed][k]) throw CudaError("event nodes missing from the step graph");
        CK(cudaGraphInstantiate(&gexec_[timed], graph, 0));
    }
    cudaGraphNode_t last_captured_node(cudaStream_t st) {
        cudaStreamCaptureStatus cs;
        const cudaGraphNode_t* deps = nullptr;
        size_t nd = 0;
        CK(cudaStreamGetCaptureInfo(st, &cs, nullptr, nullptr, &deps, &nd));
        if (nd != 1) throw CudaError("unexpected capture dependencies");
        return deps[0];
    }
    void launch_graph() {
        if (timing_) {
            cudaEvent_t* r = next_record();
            for (int k = 0; k < NMARK; k++)
                if (mark_on(timing_, k))
                    CK(cudaGraphExecEventRecordNodeSetEvent(gexec_[timing_], gev_node_[timing_][k], r[k]));
        }
        CK(cudaGraphLaunch(gexec_[timing_], stream_));
    }

    // Many steps in one graph launch: a while node whose body is k_steps (as
    // many steps as go without a rebuild) and the rebuild under an if node.
    // The step count goes to the kernel node ahead of the loop; k_steps ends
    // the loop when it has taken them, or at once when a rebuild has run out
    // of pair capacity (the host then finishes that step, as after a per-step
    // graph).  Step graphs with timing event nodes stay one step per launch
    // (an event node in a loop body would be overwritten by every iteration).
    // If the loop graph cannot be built the engine keeps launching one step
    // per graph.
    void capture_loop(Loop& l) {
        l.tried = true;
        capturing_ = true;
        capture_timed_ = 0;
        try {
            CK(cudaGraphCreate(&l.graph, 0));
            cudaGraphConditionalHandle hw;
            CK(cudaGraphConditionalHandleCreate(&hw, l.graph, 1, cudaGraphCondAssignDefault));
            CK(cudaStreamBeginCaptureToGraph(stream_, l.graph, nullptr, nullptr, 0,
                                             cudaStreamCaptureModeThreadLocal));
            k_loop_init<<<1, 1, 0, stream_>>>(h_.loop_left, h_.step_phase, h_.step_bar, h_.step_base, 1);
            CK(cudaGetLastError());
            l.init = last_captured_node(stream_);
            cudaGraph_t body = add_conditional(l.graph, hw, cudaGraphCondTypeWhile);
            cudaGraph_t g2 = nullptr;
            CK(cudaStreamEndCapture(stream_, &g2));
            cudaGraphConditionalHandle hif;
            CK(cudaGraphConditionalHandleCreate(&hif, body, 0, cudaGraphCondAssignDefault));
            CK(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
            launch_steps(hif, hw, (int)(&l - loop_));
            cudaGraph_t rbody = add_conditional(body, hif, cudaGraphCondTypeIf);
            CK(cudaStreamEndCapture(stream_, &g2));
            CK(cudaStreamBeginCaptureToGraph(stream_, rbody, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
            launch_rebuild(false);
            CK(cudaStreamEndCapture(stream_, &g2));
            CK(cudaGraphInstantiate(&l.exec, l.graph, 0));
        } catch (const CudaError&) {
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            if (cudaStreamIsCapturing(stream_, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
                cudaGraph_t g = nullptr;
                cudaStreamEndCapture(stream_, &g);
            }
            (void)cudaGetLastError();
            if (l.exec) cudaGraphExecDestroy(l.exec);
            if (l.graph) cudaGraphDestroy(l.graph);
            l.exec = nullptr;
            l.graph = nullptr;
        }
        capturing_ = false;
    }
    // Steps of one launch of k_steps at most: about 2 ms' worth.  Its blocks fill
    // an SM each, so what other streams of the process have waiting (copies and
    // kernels of other libraries, other engines) runs between two launches; 9,000
    // spheres at rest, a call of 20,000 steps: a small kernel on another stream
    // waited 186 ms without this, and waits 1.3 with it.  A launch costs 8 us (500
    // clumps, us a step: 11.5 without turns, 11.5 with 128 steps, 11.6 with 64,
    // 11.9 with 16).
    int step_turn() const { return std::max(4, std::min(128, (int)(2000.0 / (12.0 + N_ / 2500.0)))); }
    // Blocks of k_steps: one per SM at most; a smaller scene gets blocks for
    // its warps (clump pass, or about two near pairs per subsphere) at two busy
    // warps each, so that its work spreads over the SMs (2,000 spheres in FP64,
    // us a step: 2 warps 12.8, 8 warps 15.2, 16 warps 20.7).
    //
    // Launches of engines that run beside each other have to fit the GPU
    // together, or they take turns.  One of up to 2^v engines that the process has
    // stepping on the device takes 1/2^v of the SMs at most (us for a step of each
    // of eight engines: 2,000 clumps 30, 5,000 57, 12,000 145; with one block per SM
    // 80, 93, 165; separate kernels for every step 48, 66, 172).  The engines of a
    // request server, which starts them all before it waits, take a block per 32
    // warps (8 requests of 400 to 5,000 clumps: 2 warps 47.5 ms, 16 warps 32 and in
    // one process of five 44, 32 warps 32 to 34, 64 warps 38.6).
    int step_grid(int v) const {
        int per_sm = 0;
        const void* f = sphere_any_ ? (const void*)k_steps<R, true> : (const void*)k_steps<R, false>;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, ST_THREADS, 0));
        const int warps = std::max(h_.W + cdiv(S_, 32), cdiv(2LL * N_, 32));
        return std::max(1, std::min(per_sm * sm_count_ >> v, cdiv(warps, shared_gpu_ ? 32 : 2)));
    }
    void launch_steps(cudaGraphConditionalHandle hif, cudaGraphConditionalHandle hw, int v) {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(step_grid(v));
        c.blockDim = dim3(ST_THREADS);
        c.stream = stream_;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;   // the blocks wait for one another
        at[0].val.cooperative = 1;
        c.attrs = at;
        c.numAttrs = 1;
        const Dev* dp = d_;
        if (sphere_any_) CK(cudaLaunchKernelEx(&c, k_steps<R, true>, dp, hif, hw));
        else CK(cudaLaunchKernelEx(&c, k_steps<R, false>, dp, hif, hw));
    }
    // a conditional node after the capture's current dependencies; returns its body
    cudaGraph_t add_conditional(cudaGraph_t graph, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type) {
        cudaStreamCaptureStatus st;
        const cudaGraphNode_t* deps = nullptr;
        size_t ndeps = 0;
        CK(cudaStreamGetCaptureInfo(stream_, &st, nullptr, nullptr, &deps, &ndeps));
        cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
        cp.conditional.handle = h;
        cp.conditional.type = type;
        cp.conditional.size = 1;
        cudaGraphNode_t node;
        CK(cudaGraphAddNode(&node, graph, deps, ndeps, &cp));
        CK(cudaStreamUpdateCaptureDependencies(stream_, &node, 1, cudaStreamSetCaptureDependencies));
        return cp.conditional.phGraph_out[0];
    }
    void launch_loop(int n) {
        void* args[] = {&h_.loop_left, &h_.step_phase, &h_.step_bar, &h_.step_base, &n};
        cudaKernelNodeParams kp = {};
        kp.func = (void*)k_loop_init;
        kp.gridDim = dim3(1);
        kp.blockDim = dim3(1);
        kp.kernelParams = args;
        CK(cudaGraphExecKernelNodeSetParams(cur_->exec, cur_->init, &kp));
        CK(cudaGraphLaunch(cur_->exec, stream_));
    }

    // a graph launch stopped at a rebuild whose pairs did not fit: grow and
    // finish that step's rebuild and contact pass on the host path
    void recover_halt() {
        refresh_dev();
        std::vector<int> need(S_);
        copy_(need.data(), h_.need, S_ * sizeof(int), cudaMemcpyDeviceToHost);
        std::vector<SceneDyn> y = read_dyn_all();
        layout_pairs(grown_capacities(need, y));
        int zero = 0;
        copy_(h_.halt, &zero, sizeof(int), cudaMemcpyHostToDevice);
        y = read_dyn_all();
        for (auto& v : y) v.err &= ~ERR_LIST_OVERFLOW;
        copy_(h_.dyn, y.data(), S_ * sizeof(SceneDyn), cudaMemcpyHostToDevice);
        launch_rebuild(true);
        launch_contact(false);
        CK(cudaStreamSynchronize(stream_));
        steps_done_ += 1;
    }
};

EngineBase* make_engine(const std::vector<const nbc_scene_desc*>& sc, const nbc_options& opt, bool shared_gpu) {
    if (opt.precision == NBC_PREC_F64) return new EngineT<double>(sc, opt, shared_gpu);
    return new EngineT<float>(sc, opt, shared_gpu);
}

}  // namespace nbc
