#include "optional_memory.h"

#include <algorithm>
#include <condition_variable>
#include <mutex>

#include "backend.h"

namespace bc {

namespace {

constexpr int kDevices = 64;
// The library's kernels take about 20 MB when all are loaded; a pass's scratch some 10 to 100 MB, most for experts.
constexpr size_t kRoom = (size_t)256 << 20;

// One per device (devices 64 apart share one, which only makes them wait for each other).
struct Gate {
    std::mutex mutex;
    std::condition_variable changed;
    int inside = 0;             // threads inside a LaunchScope
    int outer_waiting = 0;      // threads outside that wait for `inside` to become 0; new scopes wait for them
    bool inner_waiting = false; // a thread inside that waits for the others to leave
    std::vector<ExpandedCopies*> offered;  // in the order they were offered
    std::vector<bc_backend*> backends;
    size_t unasked = 0;  // bytes that may still be allocated before the free memory is looked at again
};

Gate& gate_of(int device) {
    static Gate* gates = new Gate[kDevices];  // never destroyed: handles may be freed while the process exits
    return gates[(unsigned)device % kDevices];
}

thread_local int t_inside = -1;  // the device of this thread's LaunchScope

// Wait for everything that may read copies; false if that cannot be done now.
bool drain(Gate& gate, int device) {
    for (bc_backend* b : gate.backends) {
        if (b->device != device || !b->held_launch_scope) continue;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(b->stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return false;
        }
    }
    for (bc_backend* b : gate.backends)
        if (b->device == device && b->held_launch_scope && cudaStreamSynchronize(b->stream) != cudaSuccess) return false;
    return true;
}

}  // namespace

LaunchScope::LaunchScope(bc_backend* backend) : device_(backend->device) {
    Gate& gate = gate_of(device_);
    std::unique_lock<std::mutex> lock(gate.mutex);
    gate.changed.wait(lock, [&] { return gate.outer_waiting == 0; });
    ++gate.inside;
    t_inside = device_;
    backend->held_launch_scope = true;
}

LaunchScope::~LaunchScope() {
    Gate& gate = gate_of(device_);
    std::lock_guard<std::mutex> lock(gate.mutex);
    --gate.inside;
    t_inside = -1;
    if (gate.outer_waiting || gate.inner_waiting) gate.changed.notify_all();
}

ExpandedCopies::~ExpandedCopies() {
    if (device_ < 0) return;
    Gate& gate = gate_of(device_);
    std::lock_guard<std::mutex> lock(gate.mutex);  // another thread may be about to take them
    if (!memory_) return;
    if (offered_) gate.offered.erase(std::find(gate.offered.begin(), gate.offered.end(), this));
    cudaSetDevice(device_);
    cudaFree(memory_);
}

cudaError_t ExpandedCopies::expand(int device, cudaStream_t stream, const std::vector<k::Mat*>& mats) {
    uint64_t bytes = 0;
    for (k::Mat* m : mats) {
        if (!m->data || m->format != BC_Q4_0 || !k::half_tiles_supported(m->n_cols)) continue;
        mats_.push_back(m);
        bytes += k::half_tiles_bytes(m->n_rows, m->n_cols);
    }
    if (bytes == 0 || !k::half_tiles_fit(bytes)) return cudaSuccess;
    if (cudaMalloc(&memory_, bytes) != cudaSuccess) {
        cudaGetLastError();
        memory_ = nullptr;
        return cudaSuccess;
    }
    device_ = device;
    char* at = static_cast<char*>(memory_);
    for (k::Mat* m : mats_) {
        const cudaError_t e = k::expand_half_tiles(stream, m->data, m->scales, m->n_rows, m->n_cols, at);
        if (e != cudaSuccess) return e;
        m->half_tiles = at;
        at += k::half_tiles_bytes(m->n_rows, m->n_cols);
    }
    return cudaSuccess;
}

void ExpandedCopies::offer() {
    if (device_ < 0) return;
    Gate& gate = gate_of(device_);
    std::lock_guard<std::mutex> lock(gate.mutex);
    gate.offered.push_back(this);
    offered_ = true;
}

void ExpandedCopies::release() {
    for (k::Mat* m : mats_) m->half_tiles = nullptr;
    cudaFree(memory_);
    memory_ = nullptr;
    offered_ = false;
}

void backend_opened(bc_backend* backend) {
    Gate& gate = gate_of(backend->device);
    std::lock_guard<std::mutex> lock(gate.mutex);
    gate.backends.push_back(backend);
}

void backend_closing(bc_backend* backend) {
    Gate& gate = gate_of(backend->device);
    std::lock_guard<std::mutex> lock(gate.mutex);
    gate.backends.erase(std::remove(gate.backends.begin(), gate.backends.end(), backend), gate.backends.end());
}

bool give_back_copies(int device) {
    Gate& gate = gate_of(device);
    std::unique_lock<std::mutex> lock(gate.mutex);
    if (t_inside >= 0) {
        // Two scopes that both want memory would wait for each other: the second goes without.
        if (gate.inner_waiting) return false;
        gate.inner_waiting = true;
        gate.changed.wait(lock, [&] { return gate.inside == 1; });
        gate.inner_waiting = false;
    } else {
        ++gate.outer_waiting;
        gate.changed.wait(lock, [&] { return gate.inside == 0; });
        --gate.outer_waiting;
        gate.changed.notify_all();  // scopes that waited enter when the lock is free
    }
    auto found = std::find_if(gate.offered.begin(), gate.offered.end(), [&](ExpandedCopies* c) { return c->device_ == device && !c->pinned_; });
    if (found == gate.offered.end() || !drain(gate, device)) return false;
    ExpandedCopies* copies = *found;
    gate.offered.erase(found);
    copies->release();
    return true;
}

// Asking the driver for the free memory takes 65 us, on a busy host 600, where a whole sequence is set up in 350; so it is asked when
// what was allocated since the last time is half of what was free beyond the room then.
void keep_room(size_t bytes) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return;
    Gate& gate = gate_of(device);
    for (;;) {
        {
            std::lock_guard<std::mutex> lock(gate.mutex);
            if (gate.offered.empty()) return;
            if (bytes < gate.unasked) {
                gate.unasked -= bytes;
                return;
            }
        }
        size_t free_bytes = 0, total_bytes = 0;
        if (cudaMemGetInfo(&free_bytes, &total_bytes) != cudaSuccess) return;
        if (free_bytes >= kRoom) {
            std::lock_guard<std::mutex> lock(gate.mutex);
            gate.unasked = (free_bytes - kRoom) / 2;
            return;
        }
        if (!give_back_copies(device)) return;
    }
}

cudaError_t device_malloc(void** out, size_t bytes) {
    for (;;) {
        const cudaError_t e = cudaMalloc(out, bytes);
        if (e == cudaSuccess) {
            keep_room(bytes);
            return e;
        }
        cudaGetLastError();  // the next launch must not take this failure for its own
        *out = nullptr;
        int device = 0;
        if (e != cudaErrorMemoryAllocation || cudaGetDevice(&device) != cudaSuccess || !give_back_copies(device)) return e;
    }
}

}  // namespace bc
