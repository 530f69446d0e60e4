// Error-message plumbing for the C ABI.
#include <stdarg.h>
#include <stdio.h>

#include "us3d_common.cuh"

namespace us3d {

static thread_local char g_last_error[1024] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
    va_end(ap);
}

}  // namespace us3d

extern "C" const char* us3d_last_error(void) { return us3d::g_last_error; }

extern "C" int us3d_version(void) { return 100; }

extern "C" int us3d_set_device(int device) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        us3d::set_error("cudaSetDevice(%d) failed: %s", device, cudaGetErrorString(e));
        return US3D_CUDA_ERROR;
    }
    return US3D_OK;
}

// ---- launch counter and stage timing (benchmark instrumentation) ----
#include <atomic>
#include <mutex>
#include <new>
#include <string.h>
#include <vector>

namespace us3d {

static std::atomic<long long> g_launches{0};

void count_launches(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

struct StageProfile {
    char name[64] = {0};
    std::vector<cudaEvent_t> start, stop;
    int used = 0;
    bool enabled = false;
};

static std::mutex g_prof_mu;
static StageProfile g_prof;

// Records the "start" event of the next bracket if `name` is the profiled stage.
int prof_begin(const char* name, cudaStream_t stream) {
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (!g_prof.enabled || strcmp(name, g_prof.name) != 0 || g_prof.used >= (int)g_prof.start.size()) return -1;
    cudaEventRecord(g_prof.start[g_prof.used], stream);
    return g_prof.used++;
}

void prof_end(int slot, cudaStream_t stream) {
    if (slot < 0) return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    cudaEventRecord(g_prof.stop[slot], stream);
}

}  // namespace us3d

extern "C" long long us3d_launch_count(void) { return us3d::g_launches.load(); }

extern "C" int us3d_profile_stage(const char* stage, int max_launches) {
    std::lock_guard<std::mutex> lk(us3d::g_prof_mu);
    auto& p = us3d::g_prof;
    for (size_t i = 0; i < p.start.size(); ++i) {
        cudaEventDestroy(p.start[i]);
        cudaEventDestroy(p.stop[i]);
    }
    p.start.clear();
    p.stop.clear();
    p.used = 0;
    p.enabled = false;
    if (stage == nullptr || max_launches <= 0) return US3D_OK;
    snprintf(p.name, sizeof(p.name), "%s", stage);
    p.start.resize(max_launches);
    p.stop.resize(max_launches);
    for (int i = 0; i < max_launches; ++i) {
        if (cudaEventCreate(&p.start[i]) != cudaSuccess || cudaEventCreate(&p.stop[i]) != cudaSuccess) {
            us3d::set_error("cudaEventCreate failed");
            return US3D_CUDA_ERROR;
        }
    }
    p.enabled = true;
    return US3D_OK;
}

extern "C" int us3d_profile_collect(int* n_launches, double* total_ms) {
    std::lock_guard<std::mutex> lk(us3d::g_prof_mu);
    auto& p = us3d::g_prof;
    double tot = 0.0;
    for (int i = 0; i < p.used; ++i) {
        if (cudaEventSynchronize(p.stop[i]) != cudaSuccess) {
            us3d::set_error("cudaEventSynchronize failed");
            return US3D_CUDA_ERROR;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, p.start[i], p.stop[i]);
        tot += ms;
    }
    if (n_launches) *n_launches = p.used;
    if (total_ms) *total_ms = tot;
    p.used = 0;
    return US3D_OK;
}

// ---- status words read back to the host ----
namespace us3d {

namespace {
struct StatusSlot {
    long long* words;  // pinned
    cudaEvent_t done;
    int device;
};
constexpr int STATUS_SLOTS_KEPT = 32;  // idle slots kept; beyond that a returned slot is freed
std::mutex g_slot_mu;
StatusSlot* g_idle[STATUS_SLOTS_KEPT];
int g_n_idle = 0;

void free_slot(StatusSlot* s) {
    if (s->done) cudaEventDestroy(s->done);
    if (s->words) cudaFreeHost(s->words);
    delete s;
}

cudaError_t acquire_slot(StatusSlot** out) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lk(g_slot_mu);
        for (int i = 0; i < g_n_idle; ++i)
            if (g_idle[i]->device == device) {
                *out = g_idle[i];
                g_idle[i] = g_idle[--g_n_idle];
                return cudaSuccess;
            }
    }
    StatusSlot* s = new (std::nothrow) StatusSlot{nullptr, nullptr, device};
    if (s == nullptr) return cudaErrorMemoryAllocation;
    e = cudaHostAlloc(reinterpret_cast<void**>(&s->words), sizeof(long long) * STATUS_WORDS, cudaHostAllocPortable);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        free_slot(s);
        return e;
    }
    *out = s;
    return cudaSuccess;
}
}  // namespace

StatusRead::~StatusRead() {
    StatusSlot* s = static_cast<StatusSlot*>(slot_);
    if (s == nullptr) return;
    if (pending_) cudaEventSynchronize(s->done);  // an error return in between: the copy may still be under way
    {
        std::lock_guard<std::mutex> lk(g_slot_mu);
        if (g_n_idle < STATUS_SLOTS_KEPT) {
            g_idle[g_n_idle++] = s;
            return;
        }
    }
    free_slot(s);
}

int StatusRead::record(const long long* words, cudaStream_t stream) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    US3D_CHECK_CUDA(cudaStreamIsCapturing(stream, &capture));
    if (capture != cudaStreamCaptureStatusNone) {
        set_error("the instance total cannot be read back while the stream is being captured");
        return US3D_CUDA_ERROR;
    }
    StatusSlot* s = nullptr;
    US3D_CHECK_CUDA(acquire_slot(&s));
    slot_ = s;
    pending_ = true;
    US3D_CHECK_CUDA(cudaMemcpyAsync(s->words, words, sizeof(long long) * STATUS_WORDS, cudaMemcpyDeviceToHost, stream));
    US3D_CHECK_CUDA(cudaEventRecord(s->done, stream));
    return US3D_OK;
}

int StatusRead::wait(long long (&out)[STATUS_WORDS]) {
    StatusSlot* s = static_cast<StatusSlot*>(slot_);
    US3D_CHECK_CUDA(cudaEventSynchronize(s->done));
    pending_ = false;
    for (int i = 0; i < STATUS_WORDS; ++i) out[i] = s->words[i];
    return US3D_OK;
}

}  // namespace us3d
