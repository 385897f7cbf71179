// Device memory that the library holds but can do without: the copies of weights expanded for products of many
// tokens. They take up to half of what is free when a model is loaded, so a later allocation may find no room that it
// would have found without them; device_malloc gives them back then, owner by owner, and tries again.
//
// Launches read the copies through k::Mat::half_tiles, which host code of several threads looks at (sequences of one
// model on several backends). So a call that looks at these pointers and launches what they point to holds a LaunchScope for as
// long as it does, and giving back waits until no other thread is inside one, then for the streams of the device's backends that
// have held one, before it clears the pointers and frees the memory.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "kernels.h"

struct bc_backend;

namespace bc {

// Inside: the expanded copies stay as they are, except that an allocation of this very scope may take them. Also held while
// a step is captured, since a stream that is being captured must not be waited for. Not nested.
class LaunchScope {
  public:
    explicit LaunchScope(bc_backend* backend);
    ~LaunchScope();
    LaunchScope(const LaunchScope&) = delete;
    LaunchScope& operator=(const LaunchScope&) = delete;

  private:
    int device_;
};

// The expanded copies of one owner, a model's weights on a device or an uploaded matrix, in one allocation.
class ExpandedCopies {
  public:
    ExpandedCopies() = default;
    ~ExpandedCopies();
    ExpandedCopies(const ExpandedCopies&) = delete;
    ExpandedCopies& operator=(const ExpandedCopies&) = delete;

    // Expand these matrices when they fit (k::half_tiles_fit), on `stream`; without room they stay as they are.
    // Those that have no expanded form are passed over.
    cudaError_t expand(int device, cudaStream_t stream, const std::vector<k::Mat*>& mats);
    // From here on the copies may be given back. Call it where other threads cannot see the matrices yet, or
    // inside a LaunchScope.
    void offer();
    // Never give them back: a stream that a caller is capturing has been handed launches that read them.
    void pin() { pinned_ = true; }

  private:
    friend bool give_back_copies(int device);
    void release();

    int device_ = -1;  // set with the allocation
    void* memory_ = nullptr;
    std::vector<k::Mat*> mats_;
    bool offered_ = false, pinned_ = false;
};

// The streams on which launches that read copies may be queued.
void backend_opened(bc_backend* backend);
void backend_closing(bc_backend* backend);

// Give the copies of one owner on the device back; false if there are none to be had. Waits for other threads' launch
// scopes, and for the streams of the backends that have held one, none of which may be in capture.
bool give_back_copies(int device);

// After an allocation of `bytes` on the current device: give copies back while little room is left beside them. Kernels that are
// loaded at their first launch, graphs and scratch need some too, and the driver does not ask here first.
void keep_room(size_t bytes);

// cudaMalloc on the current device, which gives copies back while there is no room, and keeps some. A failure leaves null and no pending error.
cudaError_t device_malloc(void** out, size_t bytes);
template <typename T>
cudaError_t device_malloc(T** out, size_t bytes) {
    return device_malloc(reinterpret_cast<void**>(out), bytes);
}

}  // namespace bc
