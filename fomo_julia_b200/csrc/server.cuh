// server.cuh -- the shot server (continuous batching) and fomo_b200_run_batch.
//
// Part of fomo_b200.cu's translation unit (included after the runtime's
// internals: fail, ctx, Medium, encode_map, Launch, ...).
//
// One worker thread per server owns the CUDA streams of its launches and the
// batch loop; the servers' shots share one stream-ordered memory pool:
//   admit   queued requests, in arrival order, while their device bytes fit
//           the HBM budget (and the shot limit); allocate and upload each
//           shot, starting it at the next batch step;
//   run     K batch steps: per FD order (and up to 16 media), the step
//           records, a velocity tile launch and its band pass, a stress tile
//           launch and its band pass, per launch set of up to 12 shots
//           (step_batch.cuh); each tile launch may start beside the band
//           pass before it (programmatic dependent launch);
//           K steps are one CUDA graph replay once captured;
//   retire  shots whose nt steps are done: record the last step's receivers,
//           copy the gather to pinned memory, free the shot's memory (stream
//           ordered), and hand the gather to the caller once its copy lands.
// The host never waits for the GPU to decide what to run: shot lifetimes are
// known in steps, so chunks are planned ahead and at most two are in flight.
#pragma once

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <condition_variable>
#include <deque>
#include <map>
#include <thread>
#include <tuple>

#include "step_batch.cuh"

namespace {

using Clock = std::chrono::steady_clock;

double ms_between(Clock::time_point a, Clock::time_point b) {
    return std::chrono::duration<double, std::milli>(b - a).count();
}

inline size_t align_up(size_t n, size_t a) { return (n + a - 1) / a * a; }

// Pinned host buffers, reused by size.
class PinnedPool {
  public:
    ~PinnedPool() {
        for (auto& b : size_) cudaFreeHost(b.first);
    }
    void* take(size_t n) {
        n = std::max<size_t>(align_up(n, 4096), 4096);
        auto it = free_.lower_bound(n);
        if (it != free_.end() && it->first <= 4 * n) {
            void* p = it->second;
            free_.erase(it);
            return p;
        }
        void* p = nullptr;
        if (cudaHostAlloc(&p, n, cudaHostAllocDefault) != cudaSuccess) return nullptr;
        size_[p] = n;
        return p;
    }
    void give(void* p) {
        if (p) free_.emplace(size_[p], p);
    }

  private:
    std::multimap<size_t, void*> free_;
    std::unordered_map<void*, size_t> size_;
};

enum ReqState { kQueued = 0, kRunning = 1, kDone = 2, kFailed = 3, kCancelled = 4 };

// Buoyancy and tile descriptors of a medium for one (dtx, dtz), shared by the
// server's shots on it.
struct Resident {
    Medium* med = nullptr;
    float dtx = 0, dtz = 0;
    int iso = 0;
    float* buoy = nullptr;
    const float* b[4] = {nullptr, nullptr, nullptr, nullptr};
    CUtensorMap bmap[4];  // tile boxes of the buoyancy arrays
    CUtensorMap mod[3];   // tile boxes of lam, mu_txx, mu_txz
    int refs = 0;
    size_t bytes = 0;
};

struct Request {
    uint64_t ticket = 0;
    Medium* med = nullptr;
    int M = 0, nbc = 0, nt = 0, src_i = 0, src_j = 0, n_rec = 0, rec_kind = 0;
    float q[5] = {0, 0, 0, 0, 0};
    float a[fomo::kMaxM] = {0};
    float dtx = 0, dtz = 0;
    std::vector<float> tabs, wavelet;
    std::vector<int> cells;
    float* gather_out = nullptr;
    size_t bytes = 0;        // device bytes of the shot itself
    size_t buoy_bytes = 0;   // device bytes of its medium's buoyancy
    // Guarded by Server::mu_.
    int state = kQueued, rc = FOMO_OK;
    std::string err;
    Clock::time_point t_submit, t_admit, t_done;
    int batch_peak = 0;
    // Worker only.
    unsigned char* d_block = nullptr;
    float* d_gather = nullptr;
    Resident* res = nullptr;
    int start = 0;           // batch step of the shot's step 1
    size_t band_off = 0, tabs_off = 0, cells_off = 0, wav_off = 0, gather_off = 0;
    fomo::BatchShot vel, str;  // the shot's launch-parameter images (velocity, stress)
    fomo::MarchShot march;     // and of the fused step (all five fields of copy c to copy 1-c)
    bool fused = false;        // runs in a fused-step launch set
    CUtensorMap halo[2][5];  // halo boxes (Geo<M>) of every field of both copies
    CUtensorMap tile[2][5];  // tile boxes of every field of both copies
    void* staging = nullptr; // pinned: gather + status word
    cudaEvent_t done_ev = nullptr;
};

// Time steps per launch a batch can be told to run (a cache file's choice or
// the server's configuration): 1 = plain launches (chunks of kPlainChunk
// steps), otherwise one graph of K steps.
constexpr int kStepChoices[3] = {1, 8, 32};
// What a batch runs otherwise: graphs of 8 steps.  A replay costs a few
// microseconds, a rebuild of the graph about 0.1 ms a step, and the graphs are
// rebuilt whenever a shot joins or leaves.  Over batches of 1 to 30 shots on
// grids from 208 x 128 to 4552 x 3927, graphs of 8 steps were the fastest or
// within 1% of it (16 shots on 2108 x 908, nt 400: 135 ms at 8, 138 at 32, 161
// at 128), and timing candidates on live chunks, as the server used to, chose
// wrong often enough to cost more than it gained.
constexpr int kStepsDefault = 1;  // index in kStepChoices
constexpr int kPlainChunk = 32;
// Chains of launches side by side (enqueue_steps).  One, two and four chains:
// 24 shots on 508 x 308, nt 800, 72, 59 and 58 ms; 30 on 208 x 128, nt 2000,
// 150, 121 and 83; 20 on mixed media 134, 131 and 132; no difference where one
// set fills the device.
constexpr int kChains = 4;
constexpr int kMaxInFlight = 4096;  // shots in flight per server (launch sets <= shots)

struct TuneKey {
    int nx, nz, M, shots_log2;
    bool operator<(const TuneKey& o) const {
        return std::tie(nx, nz, M, shots_log2) < std::tie(o.nx, o.nz, o.M, o.shots_log2);
    }
};
std::mutex g_tune_mu;
std::map<TuneKey, int> g_tune;  // from the cache file: (grid, order, batch size) -> index in kStepChoices

// Optional file of choices (environment variable FOMO_B200_TUNE_CACHE,
// tune_cache_path): lines "nx nz M shots_log2 K", read when a server starts
// (lines of the single-shot kernel choice, "step ...", are skipped here).  A
// line that ends in a word notes what ran without having been chosen: it is
// not read.  Call with g_tune_mu held.
void load_tune_cache() {
    const char* path = tune_cache_path();
    if (!path) return;
    FILE* f = std::fopen(path, "r");
    if (!f) return;
    char line[256], word[16];
    int nx, nz, M, lg, K;
    while (std::fgets(line, sizeof(line), f))
        if (std::sscanf(line, "%d %d %d %d %d %15s", &nx, &nz, &M, &lg, &K, word) == 5)
            for (int c = 0; c < 3; ++c)
                if (kStepChoices[c] == K) g_tune[TuneKey{nx, nz, M, lg}] = c;
    std::fclose(f);
}

// Notes in the file, once per process and key, that the default ran.  Call with
// g_tune_mu held.
void note_default_steps(const TuneKey& k) {
    static std::set<TuneKey> noted;
    const char* path = tune_cache_path();
    if (!path || !noted.insert(k).second) return;
    if (FILE* f = std::fopen(path, "a")) {
        std::fprintf(f, "%d %d %d %d %d default\n", k.nx, k.nz, k.M, k.shots_log2, kStepChoices[kStepsDefault]);
        std::fclose(f);
    }
}

size_t batch_smem_any(int M, bool vel, int nbc, bool iso, bool fs) {
    switch (M) {
        case 1: return fomo::tiled_smem_bytes<1>(vel, nbc, iso, fs);
        case 2: return fomo::tiled_smem_bytes<2>(vel, nbc, iso, fs);
        case 3: return fomo::tiled_smem_bytes<3>(vel, nbc, iso, fs);
        case 4: return fomo::tiled_smem_bytes<4>(vel, nbc, iso, fs);
        case 5: return fomo::tiled_smem_bytes<5>(vel, nbc, iso, fs);
        case 6: return fomo::tiled_smem_bytes<6>(vel, nbc, iso, fs);
    }
    return 0;
}

template <int M>
int set_batch_smem_M(size_t v, size_t s, bool gen) {
    if (int rc = gen ? raise_smem_limit(fomo::batch_velocity_kernel<M, true>, v)
                     : raise_smem_limit(fomo::batch_velocity_kernel<M, false>, v))
        return rc;
    return gen ? raise_smem_limit(fomo::batch_stress_kernel<M, true>, s) : raise_smem_limit(fomo::batch_stress_kernel<M, false>, s);
}

int set_batch_smem(int M, size_t v, size_t s, bool gen) {
    switch (M) {
        case 1: return set_batch_smem_M<1>(v, s, gen);
        case 2: return set_batch_smem_M<2>(v, s, gen);
        case 3: return set_batch_smem_M<3>(v, s, gen);
        case 4: return set_batch_smem_M<4>(v, s, gen);
        case 5: return set_batch_smem_M<5>(v, s, gen);
        case 6: return set_batch_smem_M<6>(v, s, gen);
    }
    return fail(FOMO_EINVAL, "M=%d not supported", M);
}


// The shots of one FD order in flight: their launches of one step.
struct LaunchSet {
    int M = 0;
    std::shared_ptr<fomo::BatchVelLaunch> lv;  // kernel parameters of the velocity launches
    std::shared_ptr<fomo::BatchStrLaunch> ls;  // and of the stress launches
    int grid_v = 0, grid_s = 0, grid_b = 0;    // velocity tiles + receivers, stress tiles, band passes
    size_t smem_v = 0, smem_s = 0;
    bool gen = false;                          // some shot has generic tiles
};

// Shots of one FD order in flight that run the fused step: one launch per
// batch step.
struct MarchSet {
    int M = 0;
    std::shared_ptr<fomo::BatchMarchLaunch> L;
    int grid = 0;
};

template <int M>
int march_plan_for(int nx, int nz, int nbc, bool fs, int slots, MarchPlan* out) {
    if constexpr (M <= 4) {
        *out = march_plan<M>(nx, nz, nbc, fs, slots, g_march_segs.load());
        return FOMO_OK;
    } else {
        return FOMO_EINVAL;
    }
}

// The fused-step plan of a request's grid with `slots` blocks to fill.
MarchPlan request_march_plan(const Medium& m, int nbc, int M, int slots) {
    MarchPlan p;
    switch (M) {
        case 1: march_plan_for<1>(m.nx, m.nz, nbc, m.fs != 0, slots, &p); break;
        case 2: march_plan_for<2>(m.nx, m.nz, nbc, m.fs != 0, slots, &p); break;
        case 3: march_plan_for<3>(m.nx, m.nz, nbc, m.fs != 0, slots, &p); break;
        case 4: march_plan_for<4>(m.nx, m.nz, nbc, m.fs != 0, slots, &p); break;
    }
    return p;
}

int march_slots_of(int M) {
    switch (M) {
        case 1: return march_slots<1>();
        case 2: return march_slots<2>();
        case 3: return march_slots<3>();
        case 4: return march_slots<4>();
    }
    return 2 * sm_count();
}

size_t march_smem_bytes_any(int M) {
    switch (M) {
        case 1: return fomo::march_smem_bytes<1>();
        case 2: return fomo::march_smem_bytes<2>();
        case 3: return fomo::march_smem_bytes<3>();
        case 4: return fomo::march_smem_bytes<4>();
    }
    return 0;
}

cudaError_t batch_march_launch_any(int M, int blocks, cudaStream_t st, const fomo::BatchMarchLaunch& L) {
    switch (M) {
        case 1: return fomo::batch_march_launch<1>(blocks, st, L);
        case 2: return fomo::batch_march_launch<2>(blocks, st, L);
        case 3: return fomo::batch_march_launch<3>(blocks, st, L);
        case 4: return fomo::batch_march_launch<4>(blocks, st, L);
    }
    return cudaErrorInvalidValue;
}

const void* batch_march_kernel_any(int M) {
    switch (M) {
        case 1: return fomo::batch_march_kernel_fn<1>();
        case 2: return fomo::batch_march_kernel_fn<2>();
        case 3: return fomo::batch_march_kernel_fn<3>();
        case 4: return fomo::batch_march_kernel_fn<4>();
    }
    return nullptr;
}

// A request runs the fused step when it is selected (FOMO_STEP_FUSED) and
// supports the request's grid (M <= 4, free surface, HABC bands within its
// edge strips).
bool march_ok(const Request& r) {
    // FOMO_STEP_AUTO keeps the split launches here: measured on the batched
    // workload, the fused batch launches took 2.25x the split ones' time.
    if (g_step_mode.load() != FOMO_STEP_FUSED || r.M > 4) return false;
    return request_march_plan(*r.med, r.nbc, r.M, march_slots_of(r.M)).ok;
}

// A set's tile launch of one half step (after_band: a dependent launch
// beside the band pass just before it, see launch_tiles).
template <int M>
cudaError_t launch_batch_M(bool vel, const LaunchSet& S, cudaStream_t st, bool after_band) {
    if (vel)
        return launch_tiles(S.gen ? fomo::batch_velocity_kernel<M, true> : fomo::batch_velocity_kernel<M, false>, S.grid_v, S.smem_v, st,
                     after_band, *S.lv);
    return launch_tiles(S.gen ? fomo::batch_stress_kernel<M, true> : fomo::batch_stress_kernel<M, false>, S.grid_s, S.smem_s, st,
                        after_band, *S.ls);
}

cudaError_t launch_batch(bool vel, const LaunchSet& S, cudaStream_t st, bool after_band) {
    switch (S.M) {
        case 1: return launch_batch_M<1>(vel, S, st, after_band);
        case 2: return launch_batch_M<2>(vel, S, st, after_band);
        case 3: return launch_batch_M<3>(vel, S, st, after_band);
        case 4: return launch_batch_M<4>(vel, S, st, after_band);
        case 5: return launch_batch_M<5>(vel, S, st, after_band);
        case 6: return launch_batch_M<6>(vel, S, st, after_band);
    }
    return cudaErrorInvalidValue;
}

// Device memory of the servers' shots: one stream-ordered pool for all of
// them, kept between servers (fomo_b200_run_batch makes one for each call, and
// mapping a batch's memory anew took 7-20 ms of it, many times that on some
// hosts).  A server keeps what it has mapped, the most it held at once, while
// it lives; beyond that kServerPoolKeep bytes stay when a server is gone, until
// the library needs the memory or shuts down.  The pool orders reuse across
// the servers' streams itself, and lives as long as a server uses it.
constexpr size_t kServerPoolKeep = 2ull << 30;
struct ServerPool {
    cudaMemPool_t pool = nullptr;
    std::vector<const std::atomic<size_t>*> peaks;  // of each server on it: the most bytes it held at once
    ~ServerPool() {
        if (pool) cudaMemPoolDestroy(pool);
    }
    size_t claimed() const {
        size_t n = 0;
        for (auto* p : peaks) n += p->load();
        return n;
    }
};
struct ServerPoolSlot {
    std::mutex mu;  // guards the pool's servers too
    std::shared_ptr<ServerPool> pool;
};
ServerPoolSlot& server_pool() {
    static ServerPoolSlot& s = *new ServerPoolSlot;  // never destroyed: no CUDA call at exit
    return s;
}

// The pool for a server; *available: the free device memory and what the pool
// has mapped beyond the other servers' share.
int acquire_server_pool(int device, const std::atomic<size_t>* peak, std::shared_ptr<ServerPool>* out, size_t* available) {
    auto& S = server_pool();
    std::lock_guard<std::mutex> lk(S.mu);
    if (!S.pool) {
        auto p = std::make_shared<ServerPool>();
        cudaMemPoolProps props;
        std::memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        CUDA_TRY(cudaMemPoolCreate(&p->pool, &props));
        uint64_t keep = UINT64_MAX;
        CUDA_TRY(cudaMemPoolSetAttribute(p->pool, cudaMemPoolAttrReleaseThreshold, &keep));
        S.pool = p;
    }
    size_t fr = 0, tot = 0;
    uint64_t reserved = 0, used = 0;
    CUDA_TRY(cudaMemGetInfo(&fr, &tot));
    CUDA_TRY(cudaMemPoolGetAttribute(S.pool->pool, cudaMemPoolAttrReservedMemCurrent, &reserved));
    CUDA_TRY(cudaMemPoolGetAttribute(S.pool->pool, cudaMemPoolAttrUsedMemCurrent, &used));
    const uint64_t taken = std::max<uint64_t>(used, S.pool->claimed());
    *available = fr + (reserved > taken ? (size_t)(reserved - taken) : 0);
    S.pool->peaks.push_back(peak);
    *out = S.pool;
    return FOMO_OK;
}

void release_server_pool(std::shared_ptr<ServerPool>& p, const std::atomic<size_t>* peak) {
    auto& S = server_pool();
    std::lock_guard<std::mutex> lk(S.mu);
    p->peaks.erase(std::find(p->peaks.begin(), p->peaks.end(), peak));
    if (S.pool == p) cudaMemPoolTrimTo(p->pool, p->claimed() + kServerPoolKeep);
    p.reset();
}

// The library needs device memory: the pool gives back all but its servers' share.
void trim_server_pool() {
    auto& S = server_pool();
    std::lock_guard<std::mutex> lk(S.mu);
    if (S.pool) cudaMemPoolTrimTo(S.pool->pool, S.pool->claimed());
}

// The library shuts down: the pool goes with its last server.
void destroy_server_pool() {
    auto& S = server_pool();
    std::lock_guard<std::mutex> lk(S.mu);
    S.pool.reset();
}

class Server {
  public:
    explicit Server(const FomoServerConfig& cfg) : cfg_(cfg) {}

    int start(int device) {
        device_ = device;
        CUDA_TRY(cudaSetDevice(device));
        CUDA_TRY(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
        for (auto& q : aux_) CUDA_TRY(cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking));
        size_t available = 0;
        if (int rc = acquire_server_pool(device, &peak_, &pool_, &available)) return rc;
        CUDA_TRY(cudaMalloc(&d_ctl_, 256 + 4 * sizeof(int) * kMaxInFlight));
        d_status_ = reinterpret_cast<int*>(d_ctl_ + 128);
        d_counters_ = reinterpret_cast<int*>(d_ctl_ + 256);
        CUDA_TRY(cudaMemset(d_status_, 0, sizeof(int)));
        budget_ = cfg_.hbm_budget_bytes ? cfg_.hbm_budget_bytes : (size_t)(0.9 * (double)available);
        {
            std::lock_guard<std::mutex> lk(g_tune_mu);
            load_tune_cache();
        }
        worker_ = std::thread([this] { loop(); });
        return FOMO_OK;
    }

    ~Server() { shutdown(); }

    void shutdown() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (stopped_) return;
            stopping_ = true;
            for (auto& r : queue_) finish_locked(*r, kCancelled, FOMO_ECANCELLED, "server destroyed before the shot ran");
            queue_.clear();
        }
        cv_work_.notify_all();
        if (worker_.joinable()) worker_.join();
        cudaSetDevice(device_);
        if (st_) cudaStreamSynchronize(st_);
        for (auto& g : graphs_) cudaGraphExecDestroy(g.second);
        graphs_.clear();
        for (auto& d : deferred_) {
            if (d.exec) cudaGraphExecDestroy(d.exec);
            if (d.ev) cudaEventDestroy(d.ev);
        }
        deferred_.clear();
        for (auto e : ev_free_) cudaEventDestroy(e);
        ev_free_.clear();
        if (st_) cudaStreamSynchronize(st_);
        if (d_ctl_) cudaFree(d_ctl_);
        d_ctl_ = nullptr;
        if (pool_) release_server_pool(pool_, &peak_);
        for (auto& q : aux_) {
            if (q) cudaStreamDestroy(q);
            q = nullptr;
        }
        if (st_) cudaStreamDestroy(st_);
        st_ = nullptr;
        std::lock_guard<std::mutex> lk(mu_);
        stopped_ = true;
        cv_done_.notify_all();
    }

    int submit(std::shared_ptr<Request> r, uint64_t* ticket) {
        std::lock_guard<std::mutex> lk(mu_);
        if (stopping_) return fail(FOMO_EINVAL, "server is shutting down");
        if (!error_.empty()) return fail(FOMO_ECUDA, "server failed: %s", error_.c_str());
        if (r->bytes + r->buoy_bytes > budget_)
            return fail(FOMO_ENOMEM, "shot needs %zu device bytes, more than the server's HBM budget of %zu",
                        r->bytes + r->buoy_bytes, budget_);
        r->ticket = next_ticket_++;
        r->t_submit = Clock::now();
        reqs_[r->ticket] = r;
        queue_.push_back(r);
        stats_.submitted += 1;
        *ticket = r->ticket;
        cv_work_.notify_all();
        return FOMO_OK;
    }

    int poll(uint64_t ticket, int32_t* done) {
        std::lock_guard<std::mutex> lk(mu_);
        auto it = reqs_.find(ticket);
        if (it == reqs_.end()) return fail(FOMO_EINVAL, "unknown ticket %llu", (unsigned long long)ticket);
        const Request& r = *it->second;
        *done = r.state >= kDone ? 1 : 0;
        if (r.state >= kFailed) return fail(r.rc, "%s", r.err.c_str());
        return FOMO_OK;
    }

    int wait(uint64_t ticket, double timeout_s, FomoRequestStats* stats) {
        std::unique_lock<std::mutex> lk(mu_);
        auto it = reqs_.find(ticket);
        if (it == reqs_.end()) return fail(FOMO_EINVAL, "unknown ticket %llu", (unsigned long long)ticket);
        std::shared_ptr<Request> r = it->second;
        auto ready = [&] { return r->state >= kDone; };
        if (timeout_s < 0) {
            cv_done_.wait(lk, ready);
        } else if (!cv_done_.wait_for(lk, std::chrono::duration<double>(timeout_s), ready)) {
            return fail(FOMO_ENOTREADY, "request %llu not finished after %.3f s", (unsigned long long)ticket, timeout_s);
        }
        if (stats) {
            std::memset(stats, 0, sizeof(*stats));
            const bool admitted = r->t_admit.time_since_epoch().count() != 0;
            stats->queue_ms = admitted ? ms_between(r->t_submit, r->t_admit) : 0;
            stats->run_ms = admitted ? ms_between(r->t_admit, r->t_done) : 0;
            stats->latency_ms = ms_between(r->t_submit, r->t_done);
            stats->steps = r->state == kDone ? r->nt : 0;
            stats->batch_peak = r->batch_peak;
        }
        reqs_.erase(ticket);
        if (r->state != kDone) return fail(r->rc, "%s", r->err.c_str());
        return FOMO_OK;
    }

    int cancel(uint64_t ticket) {
        std::lock_guard<std::mutex> lk(mu_);
        auto it = reqs_.find(ticket);
        if (it == reqs_.end()) return fail(FOMO_EINVAL, "unknown ticket %llu", (unsigned long long)ticket);
        Request& r = *it->second;
        if (r.state != kQueued) return fail(FOMO_EINVAL, "request %llu is not queued", (unsigned long long)ticket);
        for (auto q = queue_.begin(); q != queue_.end(); ++q)
            if ((*q)->ticket == ticket) {
                queue_.erase(q);
                break;
            }
        finish_locked(r, kCancelled, FOMO_ECANCELLED, "request cancelled");
        return FOMO_OK;
    }

    void get_stats(FomoServerStats* s) {
        std::lock_guard<std::mutex> lk(mu_);
        *s = stats_;
    }

    cudaStream_t stream() const { return st_; }

  private:
    struct Deferred {  // released once `ev` has completed
        cudaEvent_t ev = nullptr;
        cudaGraphExec_t exec = nullptr;
        void* pinned = nullptr;
    };
    FomoServerConfig cfg_;
    int device_ = 0;
    size_t budget_ = 0;
    cudaStream_t st_ = nullptr;
    cudaStream_t aux_[kChains - 1] = {};  // the further chains' streams, idle between chunks
    std::shared_ptr<ServerPool> pool_;
    std::atomic<size_t> peak_{0};         // the most device bytes held at once
    unsigned char* d_ctl_ = nullptr;
    int* d_counters_ = nullptr;   // per launch set: velocity and stress batch step
    int* d_status_ = nullptr;
    std::thread worker_;

    std::mutex mu_;
    std::condition_variable cv_work_, cv_done_;
    std::deque<std::shared_ptr<Request>> queue_;
    std::unordered_map<uint64_t, std::shared_ptr<Request>> reqs_;
    uint64_t next_ticket_ = 1;
    bool stopping_ = false, stopped_ = false;
    std::string error_;
    FomoServerStats stats_{};

    // Worker only.
    std::vector<std::shared_ptr<Request>> active_;
    std::vector<std::shared_ptr<Request>> retiring_;
    std::map<std::tuple<Medium*, uint32_t, uint32_t>, std::unique_ptr<Resident>> resident_;
    size_t used_ = 0;
    int64_t k_host_ = 0;          // batch steps enqueued
    bool dirty_ = true;           // membership changed since the tables were built
    std::vector<LaunchSet> sets_;
    std::vector<MarchSet> msets_;  // fused-step sets (their counters follow the split sets')
    cudaError_t enqueue_err_ = cudaSuccess;
    std::map<int, cudaGraphExec_t> graphs_;  // 2K + parity of its first step -> graph of the current tables
    std::deque<cudaEvent_t> inflight_;
    std::vector<Deferred> deferred_;
    std::vector<cudaEvent_t> ev_free_;
    PinnedPool pinned_;

    // ------------------------------------------------------------ helpers
    cudaEvent_t event() {
        if (!ev_free_.empty()) {
            cudaEvent_t e = ev_free_.back();
            ev_free_.pop_back();
            return e;
        }
        cudaEvent_t e = nullptr;
        cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
        return e;
    }
    void release_event(cudaEvent_t e) { ev_free_.push_back(e); }

    static std::tuple<Medium*, uint32_t, uint32_t> res_key(const Request& r) {
        uint32_t bx, bz;
        std::memcpy(&bx, &r.dtx, 4);
        std::memcpy(&bz, &r.dtz, 4);
        return std::make_tuple(r.med, bx, bz);
    }

    void finish_locked(Request& r, int state, int rc, const std::string& msg) {
        r.state = state;
        r.rc = rc;
        r.err = msg;
        r.t_done = Clock::now();
        if (state == kDone) stats_.completed += 1;
        else if (state == kFailed) stats_.failed += 1;
        else if (state == kCancelled) stats_.cancelled += 1;
        if (r.med) {
            r.med->users.fetch_sub(1);
            r.med = nullptr;
            g_served.fetch_sub(1);
        }
        cv_done_.notify_all();
    }

    // A CUDA failure in the worker fails every request it holds and stops
    // admission; the server must then be destroyed.
    void fatal(const std::string& msg) {
        cudaStreamSynchronize(st_);
        std::lock_guard<std::mutex> lk(mu_);
        if (error_.empty()) error_ = msg.empty() ? std::string("batch loop failed") : msg;
        for (auto& r : active_) finish_locked(*r, kFailed, FOMO_ECUDA, error_);
        for (auto& r : retiring_) finish_locked(*r, kFailed, FOMO_ECUDA, error_);
        for (auto& r : queue_) finish_locked(*r, kFailed, FOMO_ECUDA, error_);
        // the pool outlives the server: give back what the shots held
        for (auto& r : active_)
            if (r->d_block) {
                cudaFreeAsync(r->d_block, st_);
                r->d_block = nullptr;
            }
        for (auto& e : resident_) cudaFreeAsync(e.second->buoy, st_);
        resident_.clear();
        used_ = 0;
        peak_.store(0);
        active_.clear();
        retiring_.clear();
        queue_.clear();
    }

    void count_launches(int64_t n) {
        std::lock_guard<std::mutex> lk(mu_);
        stats_.kernel_launches += n;
    }

    // ------------------------------------------------------------ admission
    Resident* resident_for(Request& r, int* rc) {
        *rc = FOMO_OK;
        auto key = res_key(r);
        auto it = resident_.find(key);
        if (it != resident_.end()) return it->second.get();
        auto R = std::make_unique<Resident>();
        Medium& m = *r.med;
        R->med = r.med;
        R->dtx = r.dtx;
        R->dtz = r.dtz;
        R->iso = r.dtx == r.dtz ? 1 : 0;
        const size_t plane = (size_t)m.pitch * m.nz;
        R->bytes = (R->iso ? 2 : 4) * plane * sizeof(float);
        if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&R->buoy), R->bytes, pool_->pool, st_) != cudaSuccess) {
            *rc = fail(FOMO_ENOMEM, "buoyancy allocation of %zu bytes failed", R->bytes);
            return nullptr;
        }
        if ((*rc = fill_resident(r, *R))) {
            cudaFreeAsync(R->buoy, st_);
            return nullptr;
        }
        hold(R->bytes);
        Resident* p = R.get();
        resident_.emplace(key, std::move(R));
        return p;
    }

    // Computes a medium's buoyancy arrays and encodes its tile boxes.
    int fill_resident(Request& r, Resident& R) {
        const Medium& m = *r.med;
        const size_t plane = (size_t)m.pitch * m.nz;
        float* b0 = R.buoy;
        float* b2 = R.buoy + plane;
        float* b1 = R.iso ? b0 : R.buoy + 2 * plane;
        float* b3 = R.iso ? b2 : R.buoy + 3 * plane;
        fomo::buoyancy_kernel<<<4 * sm_count(), 256, 0, st_>>>(m.arr(0), m.arr(1), r.dtx, r.dtz, plane, b0, b1, b2, b3);
        if (cudaGetLastError() != cudaSuccess) return fail(FOMO_ECUDA, "buoyancy kernel launch failed");
        count_launches(1);
        R.b[0] = b0;
        R.b[1] = b1;
        R.b[2] = b2;
        R.b[3] = b3;
        for (int q = 0; q < 4; ++q)
            if (int rc = encode_map(&R.bmap[q], R.b[q], m.nx, m.nz, m.pitch, fomo::kTX, fomo::kTZ)) return rc;
        for (int q = 0; q < 3; ++q)
            if (int rc = encode_map(&R.mod[q], m.arr(2 + q), m.nx, m.nz, m.pitch, fomo::kTX, fomo::kTZ)) return rc;
        return FOMO_OK;
    }

    // Counts device bytes as held by the server.
    void hold(size_t bytes) {
        used_ += bytes;
        if (used_ > peak_.load()) peak_.store(used_);
    }

    template <int M>
    static int build_maps(Request& r, float* const (&field)[2][5]) {
        using G = fomo::Geo<M>;
        const Medium& m = *r.med;
        for (int c = 0; c < 2; ++c)
            for (int q = 0; q < 5; ++q) {
                if (int rc = encode_map(&r.halo[c][q], field[c][q], m.nx, m.nz, m.pitch, G::BOXW, G::BOXH)) return rc;
                if (int rc = encode_map(&r.tile[c][q], field[c][q], m.nx, m.nz, m.pitch, fomo::kTX, fomo::kTZ)) return rc;
            }
        return FOMO_OK;
    }

    static int build_maps_any(Request& r, float* const (&field)[2][5]) {
        switch (r.M) {
            case 1: return build_maps<1>(r, field);
            case 2: return build_maps<2>(r, field);
            case 3: return build_maps<3>(r, field);
            case 4: return build_maps<4>(r, field);
            case 5: return build_maps<5>(r, field);
            case 6: return build_maps<6>(r, field);
        }
        return fail(FOMO_EINVAL, "M=%d not supported", r.M);
    }

    static Launch shape_of(const Request& r) {
        const Medium& m = *r.med;
        Launch L;
        L.tiles_x = (m.nx + fomo::kTX - 1) / fomo::kTX;
        L.tiles_z = (m.nz + fomo::kTZ - 1) / fomo::kTZ;
        L.x_last = std::max(0, (m.nx + 3) / 4 * 4 - fomo::kTX);
        L.n_tile = L.tiles_x * L.tiles_z;
        L.n_band = fomo::band_warp_count(m.nx);
        const bool iso = r.dtx == r.dtz;
        L.smem_v = batch_smem_any(r.M, true, r.nbc, iso, m.fs != 0);
        L.smem_s = batch_smem_any(r.M, false, r.nbc, iso, m.fs != 0);
        return L;
    }

    // Bytes of a shot's band scratch (kBandPlanes planes of nbc rows).
    static size_t band_bytes(const Request& r) { return fomo::kBandPlanes * (size_t)r.nbc * r.med->pitch * sizeof(float); }

    // Bytes of the pinned upload area of a shot.
    static size_t stage_bytes(const Request& r) {
        return align_up(r.tabs.size() * 4, 256) + align_up(r.cells.size() * 4, 256) +
               align_up(std::max<size_t>(r.wavelet.size(), 1) * 4, 256);
    }

    // Allocates and uploads an admitted shot; `stage` is pinned memory for the
    // uploads (released with the chunk that follows).
    int admit(Request& r, unsigned char* stage) {
        int rc = FOMO_OK;
        r.res = resident_for(r, &rc);
        if (!r.res) return rc;
        r.res->refs += 1;
        const Medium& m = *r.med;
        const size_t plane = (size_t)m.pitch * m.nz * sizeof(float);
        r.band_off = 10 * plane;
        r.tabs_off = r.band_off + align_up(band_bytes(r), 256);
        r.cells_off = r.tabs_off + align_up(r.tabs.size() * 4, 256);
        r.wav_off = r.cells_off + align_up(r.cells.size() * 4, 256);
        r.gather_off = r.wav_off + align_up(std::max<size_t>(r.wavelet.size(), 1) * 4, 256);
        const size_t total = r.gather_off + align_up((size_t)r.nt * r.n_rec * 4, 256);
        if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&r.d_block), total, pool_->pool, st_) != cudaSuccess)
            return fail(FOMO_ENOMEM, "shot allocation of %zu bytes failed", total);
        r.bytes = total;
        hold(total);
        unsigned char* base = r.d_block;
        CUDA_TRY(cudaMemsetAsync(base, 0, 10 * plane, st_));
        std::memcpy(stage, r.tabs.data(), r.tabs.size() * 4);
        std::memcpy(stage + (r.cells_off - r.tabs_off), r.cells.data(), r.cells.size() * 4);
        std::memcpy(stage + (r.wav_off - r.tabs_off), r.wavelet.data(), r.wavelet.size() * 4);
        CUDA_TRY(cudaMemcpyAsync(base + r.tabs_off, stage, r.gather_off - r.tabs_off, cudaMemcpyHostToDevice, st_));
        {
            std::lock_guard<std::mutex> lk(mu_);
            stats_.h2d_bytes += (int64_t)(r.gather_off - r.tabs_off);
        }
        r.d_gather = reinterpret_cast<float*>(base + r.gather_off);
        float* field[2][5];
        for (int c = 0; c < 2; ++c)
            for (int q = 0; q < 5; ++q) field[c][q] = reinterpret_cast<float*>(base + (size_t)(c * 5 + q) * plane);
        if (int e = build_maps_any(r, field)) return e;

        fomo::StepParams P;
        std::memset(&P, 0, sizeof(P));
        P.neg_zero = -0.f;
        P.nx = m.nx;
        P.nz = m.nz;
        P.pitch = m.pitch;
        P.M = m.M;
        P.pad = m.pad;
        P.nbc = r.nbc;
        P.fs = m.fs;
        P.dtx = r.dtx;
        P.dtz = r.dtz;
        for (int l = 0; l < fomo::kMaxM; ++l) P.a[l] = r.a[l];
        P.qx = r.q[0];
        P.qz = r.q[1];
        P.qt_x = r.q[2];
        P.qt_z = r.q[3];
        P.qxt = r.q[4];
        const float* tabs = reinterpret_cast<const float*>(base + r.tabs_off);
        for (int t = 0; t < 3; ++t) P.w_tab[t] = tabs + (size_t)t * (r.nbc + 2);
        P.rho_vx = m.arr(0);
        P.rho_vz = m.arr(1);
        P.lam = m.arr(2);
        P.mu_txx = m.arr(3);
        P.mu_txz = m.arr(4);
        P.src_i = r.src_i;
        P.src_j = r.src_j;
        P.nt = r.nt;
        P.n_rec = r.n_rec;
        P.rec_kind = r.rec_kind;
        P.rec_cell = reinterpret_cast<const int*>(base + r.cells_off);
        P.gather = r.d_gather;
        const Launch L = shape_of(r);
        fomo::TiledArgs T;
        std::memset(&T, 0, sizeof(T));
        for (int q = 0; q < 4; ++q) T.b[q] = r.res->b[q];
        T.iso = r.res->iso;
        T.status = d_status_;
        T.band_pre = reinterpret_cast<float*>(base + r.band_off);
        T.n_tile_blocks = L.n_tile;
        T.tiles_x = L.tiles_x;
        T.x_last = L.x_last;
        r.start = (int)(k_host_ + 1);
        for (fomo::BatchShot* S : {&r.vel, &r.str}) {
            std::memset((void*)S, 0, sizeof(*S));
            S->T = T;
            S->wavelet = reinterpret_cast<const float*>(base + r.wav_off);
            S->n_wavelet = (int)r.wavelet.size();
            S->start = r.start;
            S->nt = r.nt;
        }
        std::memset((void*)&r.march, 0, sizeof(r.march));
        r.march.wavelet = reinterpret_cast<const float*>(base + r.wav_off);
        r.march.n_wavelet = (int)r.wavelet.size();
        r.march.start = r.start;
        r.march.nt = r.nt;
        for (int c = 0; c < 2; ++c) {
            fomo::StepParams& F = r.march.P[c];
            F = P;
            for (int q = 0; q < 5; ++q) {
                F.in[q] = field[c][q];
                F.out[q] = field[1 - c][q];
            }
        }
        r.fused = march_ok(r);
        for (int c = 0; c < 2; ++c) {  // the step reads copy c, writes copy 1-c
            const int o = 1 - c;
            fomo::StepParams& V = r.vel.P[c];
            V = P;
            for (int q = 0; q < 5; ++q) V.in[q] = field[c][q];
            V.out[fomo::VX] = field[o][fomo::VX];
            V.out[fomo::VZ] = field[o][fomo::VZ];
            fomo::StepParams& S = r.str.P[c];
            S = P;
            for (int q = 0; q < 5; ++q) S.in[q] = field[c][q];
            S.in[fomo::VX] = field[o][fomo::VX];
            S.in[fomo::VZ] = field[o][fomo::VZ];
            for (int q = 2; q < 5; ++q) S.out[q] = field[o][q];
        }
        return FOMO_OK;
    }

    // ------------------------------------------------------------ tables
    int build_tables() {
        // Order: by M, then by medium (groups), then admission.
        std::vector<Request*> order, fused;
        for (auto& r : active_) (r->fused ? fused : order).push_back(r.get());
        std::stable_sort(order.begin(), order.end(), [](const Request* x, const Request* y) {
            if (x->M != y->M) return x->M < y->M;
            return x->med < y->med;
        });
        sets_.clear();
        retire_graphs();
        // One launch set per run of at most kShotsPerLaunch shots with the
        // same M; everything it needs goes into its kernel parameters.
        for (size_t i = 0; i < order.size();) {
            // the shots of an FD order in sets of equal size, so that the chains are as long as each other
            size_t run = i;
            while (run < order.size() && order[run]->M == order[i]->M) ++run;
            const size_t left = run - i, n_sets = (left + fomo::kShotsPerLaunch - 1) / fomo::kShotsPerLaunch;
            const size_t cap = (left + n_sets - 1) / n_sets;
            LaunchSet S;
            S.M = order[i]->M;
            S.lv = std::make_shared<fomo::BatchVelLaunch>();
            S.ls = std::make_shared<fomo::BatchStrLaunch>();
            std::memset((void*)S.lv.get(), 0, sizeof(fomo::BatchVelLaunch));
            std::memset((void*)S.ls.get(), 0, sizeof(fomo::BatchStrLaunch));
            fomo::BatchHead& H = S.lv->H;
            int band = 0, tile = 0, n_groups = 0;
            size_t j = i;
            while (j < order.size() && order[j]->M == S.M && n_groups < fomo::kMaxGroups &&
                   j - i < cap) {
                size_t h = j;
                while (h < order.size() && order[h]->M == S.M && order[h]->med == order[j]->med && h - i < cap) ++h;
                const Launch L = shape_of(*order[j]);
                fomo::GroupDev& G = H.groups[n_groups++];
                G.first = (int)(j - i);
                G.n = (int)(h - j);
                G.n_band = L.n_band;
                G.n_tile = L.n_tile;
                G.band_off = band;
                G.tile_off = tile;
                band += G.n * G.n_band;
                tile += G.n * G.n_tile;
                j = h;
            }
            int rec = 0;
            H.rec_off[0] = 0;
            for (size_t k = i; k < j; ++k) {
                const Request& r = *order[k];
                const size_t t = k - i;
                rec += (r.n_rec + fomo::kThreads - 1) / fomo::kThreads;
                H.rec_off[t + 1] = rec;
                const Launch L = shape_of(r);
                S.smem_v = std::max(S.smem_v, L.smem_v);
                S.smem_s = std::max(S.smem_s, L.smem_s);
                S.gen = S.gen || fomo::tiles_generic(r.med->fs != 0, r.nbc);
                S.lv->shot[t] = r.vel;
                S.ls->shot[t] = r.str;
                for (int c = 0; c < 2; ++c) {
                    for (int f = 0; f < 3; ++f) S.lv->tau[t][c][f] = r.halo[c][fomo::TXX + f];
                    for (int f = 0; f < 2; ++f) S.lv->v[t][c][f] = r.tile[c][fomo::VX + f];
                    for (int f = 0; f < 2; ++f) S.ls->v[t][c][f] = r.halo[c][fomo::VX + f];
                    for (int f = 0; f < 3; ++f) S.ls->tau[t][c][f] = r.tile[c][fomo::TXX + f];
                }
                for (int q = 0; q < 4; ++q) S.lv->b[t][q] = r.res->bmap[q];
                for (int q = 0; q < 3; ++q) S.ls->mod[t][q] = r.res->mod[q];
            }
            int* cnt = d_counters_ + 2 * sets_.size();
            H.step = cnt;
            H.advance = cnt + 1;
            H.n_shots = (int)(j - i);
            H.n_groups = n_groups;
            H.pf_ahead = fomo::prefetch_distance(sm_count());
            H.first_wave = fomo::first_wave_blocks(sm_count());
            H.total_band = band;
            H.total_tile = tile;
            S.ls->H = H;
            S.ls->H.step = cnt + 1;
            S.ls->H.advance = cnt;
            S.grid_v = tile + rec;
            S.grid_s = tile;
            S.grid_b = band;
            if (int rc = set_batch_smem(S.M, S.smem_v, S.smem_s, S.gen)) return rc;
            sets_.push_back(S);
            i = j;
        }
        if (!sets_.empty()) {  // counters of the new sets continue at the next batch step (stream ordered)
            const int n = (int)sets_.size();
            fomo::batch_counters_kernel<<<(n + 255) / 256, 256, 0, st_>>>(d_counters_, n, (int)(k_host_ + 1));
            CUDA_TRY(cudaGetLastError());
        }
        if (int rc = build_march_sets(fused)) return rc;
        dirty_ = false;
        return FOMO_OK;
    }

    // Fused-step sets: by M, then medium and HABC width (one layout per
    // group), at most kMarchShots shots and kMarchGroups groups per set.
    int build_march_sets(std::vector<Request*>& order) {
        std::stable_sort(order.begin(), order.end(), [](const Request* x, const Request* y) {
            if (x->M != y->M) return x->M < y->M;
            if (x->med != y->med) return x->med < y->med;
            return x->nbc < y->nbc;
        });
        msets_.clear();
        for (size_t i = 0; i < order.size();) {
            MarchSet S;
            S.M = order[i]->M;
            S.L = std::make_shared<fomo::BatchMarchLaunch>();
            fomo::BatchMarchLaunch& L = *S.L;
            std::memset((void*)&L, 0, sizeof(L));
            int items = 0, n_groups = 0;
            size_t j = i;
            while (j < order.size() && order[j]->M == S.M && n_groups < fomo::kMarchGroups &&
                   j - i < (size_t)fomo::kMarchShots) {
                size_t h = j;
                while (h < order.size() && order[h]->M == S.M && order[h]->med == order[j]->med &&
                       order[h]->nbc == order[j]->nbc && h - i < (size_t)fomo::kMarchShots)
                    ++h;
                const int n = (int)(h - j);
                const MarchPlan plan =
                    request_march_plan(*order[j]->med, order[j]->nbc, S.M, std::max(1, march_slots_of(S.M) / n));
                if (!plan.ok) return fail(FOMO_ECUDA, "fused-step plan lost for a running shot: %s", plan.why);
                fomo::MarchGroup& G = L.groups[n_groups++];
                G.A = plan.A;
                for (int q = 0; q < 4; ++q) G.A.b[q] = order[j]->res->b[q];
                G.A.iso = order[j]->res->iso;
                G.A.status = d_status_;
                G.first = (int)(j - i);
                G.n = n;
                G.item_off = items;
                items += n * plan.A.n_items;
                j = h;
            }
            int rec = 0;
            L.rec_off[0] = 0;
            for (size_t k = i; k < j; ++k) {
                const Request& r = *order[k];
                const size_t t = k - i;
                rec += (r.n_rec + fomo::kMThreads - 1) / fomo::kMThreads;
                L.rec_off[t + 1] = rec;
                L.shot[t] = r.march;
                for (int c = 0; c < 2; ++c)
                    for (int f = 0; f < 3; ++f) L.tau[t][c][f] = r.halo[c][fomo::TXX + f];
            }
            // counters after the split sets' (2 ints each): step, blocks left, next item, spare
            int* cnt = d_counters_ + 2 * sets_.size() + 4 * msets_.size();
            L.step = cnt;
            L.n_shots = (int)(j - i);
            L.n_groups = n_groups;
            L.total_items = items;
            L.n_rec_items = rec;
            S.grid = std::min(items + rec, march_slots_of(S.M));  // persistent blocks
            if (int rc = raise_smem_limit(batch_march_kernel_any(S.M), march_smem_bytes_any(S.M))) return rc;
            msets_.push_back(S);
            i = j;
        }
        if (!msets_.empty()) {
            const int n = (int)msets_.size();
            fomo::march_counters_kernel<<<(n + 255) / 256, 256, 0, st_>>>(d_counters_ + 2 * sets_.size(), n,
                                                                         (int)(k_host_ + 1));
            CUDA_TRY(cudaGetLastError());
        }
        return FOMO_OK;
    }

    // Graphs of the old tables are destroyed once the launches queued so far
    // are done.
    void retire_graphs() {
        for (auto& g : graphs_) {
            Deferred d;
            d.ev = event();
            d.exec = g.second;
            cudaEventRecord(d.ev, st_);
            deferred_.push_back(d);
        }
        graphs_.clear();
    }

    // ------------------------------------------------------------ stepping
    int launches_per_step() const { return 4 * (int)sets_.size() + (int)msets_.size(); }

    // `n` batch steps from step `k0` (only a step's parity goes into the
    // launches, which take it as the copy parity of their shots).  The launch
    // sets are independent of each other: they run in up to kChains chains of
    // launches side by side, set i in chain i % chains, so that one set's
    // band passes and last waves of tiles are filled by another's tiles.
    // Inside a chain every tile launch but the first follows a band pass on
    // its stream and may start beside it.  The chains fork from the server's
    // stream and join it again (in a captured graph these are its branches).
    void enqueue_steps(int n, int64_t k0) {
        const int chains = std::max(1, std::min<int>(kChains, (int)sets_.size()));
        cudaStream_t st[kChains] = {st_};
        if (chains > 1) {
            cudaEvent_t fork = event();
            note(cudaEventRecord(fork, st_));
            for (int c = 1; c < chains; ++c) {
                st[c] = aux_[c - 1];
                note(cudaStreamWaitEvent(st[c], fork, 0));
            }
            release_event(fork);
        }
        for (int k = 0; k < n; ++k) {
            for (size_t i = 0; i < sets_.size(); ++i) {
                const LaunchSet& S = sets_[i];
                cudaStream_t q = st[i % chains];
                // the step before ended with a band pass on the chain's stream, unless fused-step sets ran after it
                const bool after_band = (k > 0 && (msets_.empty() || i % chains > 0)) || i >= (size_t)chains;
                S.lv->H.kpar = S.ls->H.kpar = (int)((k0 + k) & 1);
                note(launch_batch(true, S, q, after_band));
                fomo::batch_band_kernel<true, fomo::BatchVelLaunch><<<S.grid_b, 32, 0, q>>>(*S.lv);
                note(launch_batch(false, S, q, true));
                fomo::batch_band_kernel<false, fomo::BatchStrLaunch><<<S.grid_b, 32, 0, q>>>(*S.ls);
            }
            for (const MarchSet& S : msets_) note(batch_march_launch_any(S.M, S.grid, st_, *S.L));
        }
        for (int c = 1; c < chains; ++c) {
            cudaEvent_t join = event();
            note(cudaEventRecord(join, st[c]));
            note(cudaStreamWaitEvent(st_, join, 0));
            release_event(join);
        }
    }

    // Keeps the first error of the launches enqueued since the last check.
    void note(cudaError_t e) {
        if (e != cudaSuccess && enqueue_err_ == cudaSuccess) enqueue_err_ = e;
    }

    // The first launch error since the last check.
    int take_enqueue_error() {
        const cudaError_t e = enqueue_err_;
        enqueue_err_ = cudaSuccess;
        if (e != cudaSuccess) return fail(FOMO_ECUDA, "batch launch failed: %s", cudaGetErrorString(e));
        return FOMO_OK;
    }

    // The graph of K batch steps starting at a step of parity p0.
    int graph_for(int K, int p0, cudaGraphExec_t* out) {
        const int key = 2 * K + p0;
        auto it = graphs_.find(key);
        if (it != graphs_.end()) {
            *out = it->second;
            return FOMO_OK;
        }
        cudaGraph_t g = nullptr;
        CUDA_TRY(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
        enqueue_steps(K, p0);
        cudaError_t e = cudaStreamEndCapture(st_, &g);
        if (int rc = take_enqueue_error()) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (e != cudaSuccess) return fail(FOMO_ECUDA, "graph capture failed: %s", cudaGetErrorString(e));
        cudaGraphExec_t x = nullptr;
        e = cudaGraphInstantiate(&x, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return fail(FOMO_ECUDA, "graph instantiation failed: %s", cudaGetErrorString(e));
        // upload now, so that the first replay does not carry it
        e = cudaGraphUpload(x, st_);
        if (e != cudaSuccess) return fail(FOMO_ECUDA, "graph upload failed: %s", cudaGetErrorString(e));
        graphs_[key] = x;
        *out = x;
        return FOMO_OK;
    }

    TuneKey tune_key() const {
        // The largest medium in flight names the batch.
        const Request* big = active_.front().get();
        for (auto& r : active_)
            if ((double)r->med->nx * r->med->nz > (double)big->med->nx * big->med->nz) big = r.get();
        int n = (int)active_.size(), lg = 0;
        while ((1 << (lg + 1)) <= n) ++lg;
        return TuneKey{big->med->nx, big->med->nz, big->M, lg};
    }

    // Index in kStepChoices of the next chunk (-2: a configured K that is none
    // of them): the configuration's, the cache file's, or the default.
    int choose(const TuneKey& key) {
        if (cfg_.steps_per_launch > 0) {
            for (int c = 0; c < 3; ++c)
                if (kStepChoices[c] == cfg_.steps_per_launch) return c;
            return -2;
        }
        std::lock_guard<std::mutex> lk(g_tune_mu);
        const auto it = g_tune.find(key);
        if (it != g_tune.end()) return it->second;
        note_default_steps(key);
        return kStepsDefault;
    }

    int run_chunk() {
        int64_t rem = INT64_MAX;
        for (auto& r : active_) rem = std::min<int64_t>(rem, (int64_t)r->start + r->nt - 1 - k_host_);
        const int cand = choose(tune_key());
        const int K = cand >= 0 ? kStepChoices[cand] : cfg_.steps_per_launch;
        const int chunk = K == 1 ? kPlainChunk : K;
        const int n = (int)std::min<int64_t>(chunk, rem);
        const bool graph = K > 1 && n == K;
        cudaGraphExec_t x = nullptr;
        if (graph)
            if (int rc = graph_for(K, (int)((k_host_ + 1) & 1), &x)) return rc;
        nvtxRangePushA(graph ? "fomo_b200 batch graph replay" : "fomo_b200 batch launches");
        if (graph) {
            const cudaError_t e = cudaGraphLaunch(x, st_);
            nvtxRangePop();
            CUDA_TRY(e);
        } else {
            enqueue_steps(n, k_host_ + 1);
            nvtxRangePop();
            CUDA_TRY(cudaGetLastError());
            if (int rc = take_enqueue_error()) return rc;
        }
        k_host_ += n;
        {
            std::lock_guard<std::mutex> lk(mu_);
            stats_.batch_steps += n;
            stats_.kernel_launches += (int64_t)n * launches_per_step();
            if (graph) stats_.graph_replays += 1;
            stats_.steps_per_launch = graph ? K : 1;
            const int na = (int)active_.size();
            for (auto& r : active_) r->batch_peak = std::max(r->batch_peak, na);
        }
        cudaEvent_t e = event();
        CUDA_TRY(cudaEventRecord(e, st_));
        inflight_.push_back(e);
        return FOMO_OK;
    }

    // ------------------------------------------------------------ retirement
    int retire_done() {
        bool any = false;
        for (size_t i = 0; i < active_.size();) {
            Request& r = *active_[i];
            if ((int64_t)r.start + r.nt - 1 > k_host_) {
                ++i;
                continue;
            }
            if (int rc = retire(r)) return rc;
            retiring_.push_back(active_[i]);
            active_.erase(active_.begin() + i);
            any = true;
        }
        if (any) dirty_ = true;
        return FOMO_OK;
    }

    int retire(Request& r) {
        const size_t gbytes = (size_t)r.nt * r.n_rec * sizeof(float);
        if (r.n_rec > 0 && r.nt > 0) {  // receivers of the last step
            fomo::StepParams P = r.vel.P[r.nt & 1];  // reads copy nt & 1: the state after step nt
            P.rec_k = r.nt;
            fomo::record_kernel<<<(r.n_rec + fomo::kThreads - 1) / fomo::kThreads, fomo::kThreads, 0, st_>>>(P);
            CUDA_TRY(cudaGetLastError());
            count_launches(1);
        }
        r.staging = pinned_.take(gbytes + 16);
        if (!r.staging) return fail(FOMO_ENOMEM, "pinned staging of %zu bytes failed", gbytes + 16);
        if (gbytes) CUDA_TRY(cudaMemcpyAsync(r.staging, r.d_gather, gbytes, cudaMemcpyDeviceToHost, st_));
        CUDA_TRY(cudaMemcpyAsync(static_cast<unsigned char*>(r.staging) + align_up(gbytes, 16), d_status_, sizeof(int),
                                 cudaMemcpyDeviceToHost, st_));
        CUDA_TRY(cudaFreeAsync(r.d_block, st_));
        r.d_block = nullptr;
        r.done_ev = event();
        CUDA_TRY(cudaEventRecord(r.done_ev, st_));
        used_ -= r.bytes;
        Resident* R = r.res;
        r.res = nullptr;
        if (R && --R->refs == 0) {
            CUDA_TRY(cudaFreeAsync(R->buoy, st_));
            used_ -= R->bytes;
            for (auto it = resident_.begin(); it != resident_.end(); ++it)
                if (it->second.get() == R) {
                    resident_.erase(it);
                    break;
                }
        }
        std::lock_guard<std::mutex> lk(mu_);
        stats_.d2h_bytes += (int64_t)gbytes;
        return FOMO_OK;
    }

    // Hands over the gathers whose copies have landed.
    void complete_retired(bool block) {
        for (size_t i = 0; i < retiring_.size();) {
            Request& r = *retiring_[i];
            if (block) cudaEventSynchronize(r.done_ev);
            if (cudaEventQuery(r.done_ev) != cudaSuccess) {
                ++i;
                continue;
            }
            const size_t gbytes = (size_t)r.nt * r.n_rec * sizeof(float);
            int status = 0;
            std::memcpy(&status, static_cast<unsigned char*>(r.staging) + align_up(gbytes, 16), sizeof(int));
            if (!status && gbytes) std::memcpy(r.gather_out, r.staging, gbytes);
            pinned_.give(r.staging);
            r.staging = nullptr;
            release_event(r.done_ev);
            r.done_ev = nullptr;
            {
                std::lock_guard<std::mutex> lk(mu_);
                if (status == fomo::kErrTmaTimeout)
                    finish_locked(r, kFailed, FOMO_ETIMEOUT, "a TMA load of a batch time-step kernel did not complete");
                else if (status == fomo::kErrBatchParity)
                    finish_locked(r, kFailed, FOMO_ECUDA, "a batch launch's step parity disagreed with its step counter");
                else if (status)
                    finish_locked(r, kFailed, FOMO_ECUDA, "batch time-step kernel reported error " + std::to_string(status));
                else
                    finish_locked(r, kDone, FOMO_OK, "");
            }
            retiring_.erase(retiring_.begin() + i);
        }
    }

    void release_deferred(bool block) {
        for (size_t i = 0; i < deferred_.size();) {
            Deferred& d = deferred_[i];
            if (block) cudaEventSynchronize(d.ev);
            if (cudaEventQuery(d.ev) != cudaSuccess) {
                ++i;
                continue;
            }
            if (d.exec) cudaGraphExecDestroy(d.exec);
            if (d.pinned) pinned_.give(d.pinned);
            release_event(d.ev);
            deferred_.erase(deferred_.begin() + i);
        }
    }

    // ------------------------------------------------------------ the loop
    void loop() {
        cudaSetDevice(device_);
        while (true) {
            complete_retired(false);
            release_deferred(false);
            std::vector<std::shared_ptr<Request>> admitted;
            {
                std::unique_lock<std::mutex> lk(mu_);
                if (active_.empty() && queue_.empty()) {
                    if (stopping_ && retiring_.empty()) break;
                    if (retiring_.empty() && deferred_.empty()) {
                        cv_work_.wait(lk, [&] { return stopping_ || !queue_.empty(); });
                        continue;
                    }
                }
                size_t planned = used_;
                std::vector<std::tuple<Medium*, uint32_t, uint32_t>> new_res;
                while (!queue_.empty()) {
                    Request& r = *queue_.front();
                    if (cfg_.max_shots > 0 && (int)(active_.size() + admitted.size()) >= cfg_.max_shots) break;
                    if (active_.size() + admitted.size() >= (size_t)kMaxInFlight) break;
                    auto key = res_key(r);
                    const bool have = resident_.count(key) != 0 ||
                                      std::find(new_res.begin(), new_res.end(), key) != new_res.end();
                    const size_t need = r.bytes + (have ? 0 : r.buoy_bytes);
                    if (planned + need > budget_) break;
                    planned += need;
                    if (!have) new_res.push_back(key);
                    r.state = kRunning;
                    r.t_admit = Clock::now();
                    admitted.push_back(queue_.front());
                    queue_.pop_front();
                }
            }
            if (!admitted.empty()) {
                size_t sb = 0;
                for (auto& r : admitted) sb += stage_bytes(*r);
                unsigned char* stage = static_cast<unsigned char*>(pinned_.take(sb));
                if (!stage) {
                    for (auto& r : admitted) active_.push_back(r);
                    fatal("pinned staging allocation failed");
                    continue;
                }
                size_t off = 0;
                int rc = FOMO_OK;
                size_t k = 0;
                for (; k < admitted.size(); ++k) {
                    auto& r = admitted[k];
                    if (r->nt == 0) {  // nothing to run: done at once
                        std::lock_guard<std::mutex> lk(mu_);
                        finish_locked(*r, kDone, FOMO_OK, "");
                        continue;
                    }
                    active_.push_back(r);
                    if ((rc = admit(*r, stage + off))) break;
                    off += stage_bytes(*r);
                    dirty_ = true;
                }
                Deferred d;
                d.ev = event();
                d.pinned = stage;
                cudaEventRecord(d.ev, st_);
                deferred_.push_back(d);
                if (rc) {
                    for (++k; k < admitted.size(); ++k) active_.push_back(admitted[k]);
                    fatal(g_err);
                    continue;
                }
                std::lock_guard<std::mutex> lk(mu_);
                stats_.peak_shots = std::max<int32_t>(stats_.peak_shots, (int32_t)active_.size());
                stats_.peak_bytes = std::max<uint64_t>(stats_.peak_bytes, used_);
            }
            if (active_.empty()) {
                // Nothing to run: wait for copies in flight, then look again.
                if (!retiring_.empty()) complete_retired(true);
                else if (!deferred_.empty()) release_deferred(true);
                continue;
            }
            if (dirty_ && build_tables()) {
                fatal(g_err);
                continue;
            }
            if (run_chunk() || retire_done()) {
                fatal(g_err);
                continue;
            }
            while (inflight_.size() > 2) {
                cudaEventSynchronize(inflight_.front());
                release_event(inflight_.front());
                inflight_.pop_front();
            }
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) fatal(std::string("CUDA error in the batch loop: ") + cudaGetErrorString(e));
        }
        for (auto e : inflight_) {
            cudaEventSynchronize(e);
            release_event(e);
        }
        inflight_.clear();
        release_deferred(true);
    }
};

struct ServerTable {
    std::mutex mu;
    std::unordered_map<uint64_t, std::shared_ptr<Server>> servers;
    uint64_t next = 1;
};

ServerTable& servers() {
    static ServerTable t;
    return t;
}

void shutdown_servers() {
    std::vector<std::shared_ptr<Server>> all;
    {
        auto& T = servers();
        std::lock_guard<std::mutex> lk(T.mu);
        for (auto& kv : T.servers) all.push_back(kv.second);
        T.servers.clear();
    }
    for (auto& s : all) s->shutdown();
}

std::shared_ptr<Server> find_server(uint64_t h) {
    auto& T = servers();
    std::lock_guard<std::mutex> lk(T.mu);
    auto it = T.servers.find(h);
    return it == T.servers.end() ? nullptr : it->second;
}

// Validates a shot against its medium (the checks of fomo_b200_shot_begin)
// and copies it into a request.
int make_request(Medium* m, const FomoHabc* habc, const FomoShot* shot, float* gather_out,
                 std::shared_ptr<Request>* out) {
    if (!habc || !shot) return fail(FOMO_EINVAL, "NULL argument");
    if (shot->M != m->M) return fail(FOMO_EINVAL, "shot M=%d differs from medium M=%d", shot->M, m->M);
    if (!shot->a) return fail(FOMO_EINVAL, "FD coefficients are NULL");
    if (shot->nt < 0) return fail(FOMO_EINVAL, "nt=%d < 0", shot->nt);
    const int nbc = habc->nbc;
    if (int rc = check_band(m->nx, m->nz, m->pad, m->fs, nbc)) return rc;
    if (!habc->w_vx || !habc->w_vz || !habc->w_tau) return fail(FOMO_EINVAL, "HABC weight tables are NULL");
    if (shot->src_i < 1 || shot->src_i > m->nx || shot->src_j < 1 || shot->src_j > m->nz)
        return fail(FOMO_EINVAL, "source (%d, %d) outside the %dx%d grid", shot->src_i, shot->src_j, m->nx, m->nz);
    if (shot->n_wavelet < 0 || (shot->n_wavelet > 0 && !shot->wavelet)) return fail(FOMO_EINVAL, "bad wavelet");
    if (shot->n_rec < 0 || (shot->n_rec > 0 && (!shot->rec_i || !shot->rec_j)))
        return fail(FOMO_EINVAL, "bad receiver arrays");
    if (shot->rec_kind < 0 || shot->rec_kind > 2) return fail(FOMO_EINVAL, "bad receiver kind %d", shot->rec_kind);
    if (shot->n_rec > 0 && shot->nt > 0 && !gather_out) return fail(FOMO_EINVAL, "gather_out is NULL");
    const bool iso = shot->dtx == shot->dtz;
    const size_t smem = std::max(batch_smem_any(m->M, true, nbc, iso, m->fs != 0), batch_smem_any(m->M, false, nbc, iso, m->fs != 0));
    if (smem > 227 * 1024)
        return fail(FOMO_EINVAL, "nbc=%d needs %zu bytes of shared memory per block, more than 227 KB", nbc, smem);
    auto r = std::make_shared<Request>();
    r->med = m;
    r->M = shot->M;
    r->nbc = nbc;
    r->nt = shot->nt;
    r->src_i = shot->src_i - 1;
    r->src_j = shot->src_j - 1;
    r->n_rec = shot->n_rec;
    r->rec_kind = shot->rec_kind;
    r->q[0] = habc->qx;
    r->q[1] = habc->qz;
    r->q[2] = habc->qt_x;
    r->q[3] = habc->qt_z;
    r->q[4] = habc->qxt;
    for (int l = 0; l < shot->M; ++l) r->a[l] = shot->a[l];
    r->dtx = shot->dtx;
    r->dtz = shot->dtz;
    const size_t tab_n = (size_t)nbc + 2;
    r->tabs.resize(3 * tab_n);
    std::memcpy(r->tabs.data(), habc->w_vx, tab_n * 4);
    std::memcpy(r->tabs.data() + tab_n, habc->w_vz, tab_n * 4);
    std::memcpy(r->tabs.data() + 2 * tab_n, habc->w_tau, tab_n * 4);
    r->wavelet.assign(shot->wavelet, shot->wavelet + shot->n_wavelet);
    r->cells.resize(shot->n_rec);
    for (int k = 0; k < shot->n_rec; ++k) {
        const int i = shot->rec_i[k], j = shot->rec_j[k];
        if (i < 1 || i > m->nx || j < 1 || j > m->nz)
            return fail(FOMO_EINVAL, "receiver %d at (%d, %d) outside the %dx%d grid", k + 1, i, j, m->nx, m->nz);
        r->cells[k] = (i - 1) + (j - 1) * m->pitch;
    }
    r->gather_out = gather_out;
    const size_t plane = (size_t)m->pitch * m->nz * sizeof(float);
    r->bytes = 10 * plane + align_up(fomo::kBandPlanes * (size_t)nbc * m->pitch * sizeof(float), 256) + align_up(r->tabs.size() * 4, 256) + align_up(r->cells.size() * 4, 256) +
               align_up(std::max<size_t>(r->wavelet.size(), 1) * 4, 256) +
               align_up((size_t)r->nt * r->n_rec * 4, 256);
    r->buoy_bytes = (iso ? 2 : 4) * plane;
    *out = std::move(r);
    return FOMO_OK;
}

}  // namespace

extern "C" {

int fomo_b200_server_create(const FomoServerConfig* config, uint64_t* server) {
    int device = 0;
    {
        std::lock_guard<std::mutex> lk(ctx().mu);
        if (int rc = ensure_init()) return rc;
        device = ctx().device;
    }
    if (!server) return fail(FOMO_EINVAL, "server is NULL");
    FomoServerConfig cfg{};
    if (config) cfg = *config;
    if (cfg.max_shots < 0 || cfg.steps_per_launch < 0 || cfg.steps_per_launch > 1024)
        return fail(FOMO_EINVAL, "bad server configuration");
    auto s = std::make_shared<Server>(cfg);
    if (int rc = s->start(device)) return rc;
    auto& T = servers();
    std::lock_guard<std::mutex> lk(T.mu);
    const uint64_t h = T.next++;
    T.servers[h] = s;
    *server = h;
    return FOMO_OK;
}

int fomo_b200_server_submit(uint64_t server, uint64_t medium, const FomoHabc* habc, const FomoShot* shot,
                            float* gather_out, uint64_t* ticket) {
    auto s = find_server(server);
    if (!s) return fail(FOMO_EINVAL, "unknown server handle %llu", (unsigned long long)server);
    if (!ticket) return fail(FOMO_EINVAL, "ticket is NULL");
    std::shared_ptr<Request> r;
    {
        std::lock_guard<std::mutex> lk(ctx().mu);
        if (int rc = ensure_init()) return rc;
        Medium* m = get<Medium>(medium);
        if (!m) return fail(FOMO_EINVAL, "unknown medium handle %llu", (unsigned long long)medium);
        if (int rc = make_request(m, habc, shot, gather_out, &r)) return rc;
        m->users.fetch_add(1);
        g_served.fetch_add(1);
    }
    if (int rc = s->submit(r, ticket)) {
        r->med->users.fetch_sub(1);
        g_served.fetch_sub(1);
        return rc;
    }
    return FOMO_OK;
}

int fomo_b200_server_poll(uint64_t server, uint64_t ticket, int32_t* done) {
    auto s = find_server(server);
    if (!s) return fail(FOMO_EINVAL, "unknown server handle %llu", (unsigned long long)server);
    if (!done) return fail(FOMO_EINVAL, "done is NULL");
    return s->poll(ticket, done);
}

int fomo_b200_server_wait(uint64_t server, uint64_t ticket, double timeout_s, FomoRequestStats* stats) {
    auto s = find_server(server);
    if (!s) return fail(FOMO_EINVAL, "unknown server handle %llu", (unsigned long long)server);
    return s->wait(ticket, timeout_s, stats);
}

int fomo_b200_server_cancel(uint64_t server, uint64_t ticket) {
    auto s = find_server(server);
    if (!s) return fail(FOMO_EINVAL, "unknown server handle %llu", (unsigned long long)server);
    return s->cancel(ticket);
}

int fomo_b200_server_stats(uint64_t server, FomoServerStats* stats) {
    auto s = find_server(server);
    if (!s) return fail(FOMO_EINVAL, "unknown server handle %llu", (unsigned long long)server);
    if (!stats) return fail(FOMO_EINVAL, "stats is NULL");
    s->get_stats(stats);
    return FOMO_OK;
}

int fomo_b200_server_destroy(uint64_t server) {
    std::shared_ptr<Server> s;
    {
        auto& T = servers();
        std::lock_guard<std::mutex> lk(T.mu);
        auto it = T.servers.find(server);
        if (it == T.servers.end()) return fail(FOMO_EINVAL, "unknown server handle %llu", (unsigned long long)server);
        s = it->second;
        T.servers.erase(it);
    }
    s->shutdown();
    return FOMO_OK;
}

int fomo_b200_run_batch(uint64_t medium, const FomoHabc* habc, const FomoShot* shots, int32_t n_shots,
                        float* const* gathers_out, FomoRunStats* stats) {
    if (n_shots < 0 || (n_shots > 0 && (!shots || !gathers_out))) return fail(FOMO_EINVAL, "bad shot arrays");
    {
        std::lock_guard<std::mutex> lk(ctx().mu);
        if (int rc = ensure_init()) return rc;
        if (!get<Medium>(medium)) return fail(FOMO_EINVAL, "unknown medium handle %llu", (unsigned long long)medium);
        for (int s = 0; s < n_shots; ++s)
            if (shots[s].dtx != shots[0].dtx || shots[s].dtz != shots[0].dtz)
                return fail(FOMO_EINVAL, "shot %d has dtx/dtz different from shot 0's", s);
    }
    uint64_t h = 0;
    FomoServerConfig cfg{};
    if (int rc = fomo_b200_server_create(&cfg, &h)) return rc;
    auto srv = find_server(h);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, srv->stream());
    std::vector<uint64_t> tickets;
    int rc = FOMO_OK;
    for (int s = 0; s < n_shots && rc == FOMO_OK; ++s) {
        uint64_t t = 0;
        rc = fomo_b200_server_submit(h, medium, habc, &shots[s], gathers_out[s], &t);
        if (rc == FOMO_OK) tickets.push_back(t);
    }
    std::string msg = rc ? g_err : std::string();
    int64_t steps = 0;
    for (uint64_t t : tickets) {
        FomoRequestStats rs;
        std::memset(&rs, 0, sizeof(rs));
        const int w = fomo_b200_server_wait(h, t, -1.0, &rs);
        if (w && rc == FOMO_OK) {
            rc = w;
            msg = g_err;
        }
        steps += rs.steps;
    }
    cudaEventRecord(e1, srv->stream());
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    FomoServerStats ss;
    srv->get_stats(&ss);
    srv.reset();
    fomo_b200_server_destroy(h);
    if (stats) {
        stats->device_ms = ms;
        stats->steps = steps;
        stats->kernel_launches = ss.kernel_launches;
        stats->h2d_bytes = ss.h2d_bytes;
        stats->d2h_bytes = ss.d2h_bytes;
    }
    if (rc) g_err = msg;
    return rc;
}

}  // extern "C"
