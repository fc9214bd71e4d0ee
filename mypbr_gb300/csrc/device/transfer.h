// Copies of frames between pageable host memory and the GPU, and device
// workspaces that calls without a scene handle reuse.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace mypbr_dev {

// Copies that are done when they return, each ordered as one transfer on its
// stream (to the device: the legacy stream). The pages of a new frame are made
// before it is written.
int copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st);
int copy_to_device(void* dst, const void* src, size_t bytes);

// Device memory for one call on the current device, taken apart in pieces
// (256-byte aligned). The bytes asked for first come from a workspace that is
// kept for the next call; while another thread uses it, or past
// kWorkspaceMost, the memory is the call's own. The caller's work on it has to
// be done before the object goes.
class Workspace {
  public:
    Workspace() = default;
    ~Workspace();
    Workspace(const Workspace&) = delete;
    Workspace& operator=(const Workspace&) = delete;
    int reserve(size_t bytes);
    template <typename T>
    T* take(size_t n) {
        T* p = reinterpret_cast<T*>(base_ + used_);
        used_ += padded<T>(n);
        return p;
    }
    template <typename T>
    static size_t padded(size_t n) {
        return (n * sizeof(T) + 255) / 256 * 256;
    }

  private:
    char* base_ = nullptr;
    size_t used_ = 0;
    int kept_ = -1;  // the device whose kept workspace this is, or -1: the call's own memory
};

// A zeroed int in pinned memory that kernels of every device can write, for the
// few words that a host reads after each call: reading one where it lies takes
// no transfer (4 bytes into pageable memory: 10 to 25 us of a call). Taken from
// blocks of 64 KiB (pinning one costs 0.3 ms); null when there is no memory.
int* take_host_word();
void give_host_word(int* word);

// Gives the current device's kept workspace back, if no call uses it.
void release_workspaces();

// cudaMalloc for everything but that workspace: where memory has run out the
// workspace is given back and the allocation tried again.
cudaError_t device_malloc_bytes(void** p, size_t bytes);
template <typename T>
cudaError_t device_malloc(T** p, size_t bytes) {
    return device_malloc_bytes(reinterpret_cast<void**>(p), bytes);
}

}  // namespace mypbr_dev
