// See transfer.h.
#include "transfer.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "gpu_scene.h"

namespace mypbr_dev {
namespace {

constexpr int kMaxDevices = 64;

// A pageable copy by the driver is one thread's: it stages, copies and, on a
// frame the caller has just allocated, takes every page fault (853 x 479 x 10
// doubles into fresh pages took most of 15 ms). Each thread here copies its own
// part of the frame through two pinned buffers of its own, the next transfer
// under way while it copies the last one out.
constexpr int kThreads = 8;
constexpr size_t kSlot = size_t(1) << 20;
constexpr size_t kSplitFrom = size_t(2) << 20;  // below, starting threads costs more than it saves

struct Lane {
    char* slot[2] = {nullptr, nullptr};
    cudaStream_t stream = nullptr;
    cudaEvent_t done[2] = {nullptr, nullptr};
};
struct Lanes {
    std::mutex busy;
    bool ready = false, failed = false;
    Lane lane[kThreads];
};
Lanes g_lanes[kMaxDevices];  // 16 MiB of pinned memory on each device that copies large frames

// The lanes of the current device, made by the first large copy. Called with
// their mutex held; false when they cannot be made.
bool ready(Lanes& L) {
    if (L.ready || L.failed)
        return L.ready;
    bool ok = true;
    for (Lane& l : L.lane) {
        for (int k = 0; k < 2 && ok; k++)
            ok = cudaHostAlloc(reinterpret_cast<void**>(&l.slot[k]), kSlot, cudaHostAllocDefault) == cudaSuccess &&
                 cudaEventCreateWithFlags(&l.done[k], cudaEventDisableTiming) == cudaSuccess;
        ok = ok && cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        L.failed = true;
    }
    return L.ready = ok;
}

// One thread's part of a copy, chunk by chunk. Nothing is under way on its
// stream when it returns.
cudaError_t copy_part(Lane& l, char* dst, const char* src, size_t bytes, bool to_host) {
    cudaError_t e = cudaSuccess;
    const size_t chunks = (bytes + kSlot - 1) / kSlot;
    auto length = [&](size_t c) { return std::min(kSlot, bytes - c * kSlot); };
    for (size_t c = 0; c <= chunks && e == cudaSuccess; c++) {
        if (to_host) {
            if (c < chunks) {
                e = cudaMemcpyAsync(l.slot[c & 1], src + c * kSlot, length(c), cudaMemcpyDeviceToHost, l.stream);
                if (e == cudaSuccess)
                    e = cudaEventRecord(l.done[c & 1], l.stream);
            }
            if (c > 0 && e == cudaSuccess) {
                e = cudaEventSynchronize(l.done[(c - 1) & 1]);
                if (e == cudaSuccess)
                    std::memcpy(dst + (c - 1) * kSlot, l.slot[(c - 1) & 1], length(c - 1));
            }
        } else if (c < chunks) {
            if (c >= 2)
                e = cudaEventSynchronize(l.done[c & 1]);
            if (e == cudaSuccess) {
                std::memcpy(l.slot[c & 1], src + c * kSlot, length(c));
                e = cudaMemcpyAsync(dst + c * kSlot, l.slot[c & 1], length(c), cudaMemcpyHostToDevice, l.stream);
            }
            if (e == cudaSuccess)
                e = cudaEventRecord(l.done[c & 1], l.stream);
        }
    }
    const cudaError_t last = cudaStreamSynchronize(l.stream);
    return e != cudaSuccess ? e : last;
}

// st carries the copies that are not split, after its work.
int copy(void* dst, const void* src, size_t bytes, bool to_host, cudaStream_t st) {
    int device = 0;
    MYPBR_CUDA(cudaGetDevice(&device));
    const int threads = std::min<int>(kThreads, int(std::max(1u, std::thread::hardware_concurrency())));
    if (bytes >= kSplitFrom && threads > 1 && device < kMaxDevices) {
        Lanes& L = g_lanes[device];
        std::unique_lock<std::mutex> lock(L.busy, std::try_to_lock);
        if (lock.owns_lock() && ready(L)) {
            const size_t part = (bytes / size_t(threads) + 4095) / 4096 * 4096;
            std::vector<cudaError_t> status(size_t(threads), cudaSuccess);
            auto run = [&](int t) {
                const size_t at = std::min(bytes, part * size_t(t));
                const size_t n = t == threads - 1 ? bytes - at : std::min(part, bytes - at);
                cudaError_t e = cudaSetDevice(device);
                if (e == cudaSuccess && n > 0)
                    e = copy_part(L.lane[t], static_cast<char*>(dst) + at, static_cast<const char*>(src) + at, n,
                                  to_host);
                status[size_t(t)] = e;
            };
            std::vector<std::thread> pool;
            int started = 1;
            try {
                for (; started < threads; started++)
                    pool.emplace_back(run, started);
            } catch (...) {  // no more threads to be had: this one copies the other parts too
            }
            run(0);
            for (int t = started; t < threads; t++)
                run(t);
            for (std::thread& t : pool)
                t.join();
            for (cudaError_t e : status)
                if (e != cudaSuccess)
                    return cuda_fail(e, "frame copy");
            return MYPBR_OK;
        }
    }
    MYPBR_CUDA(cudaMemcpyAsync(dst, src, bytes, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st));
    MYPBR_CUDA(cudaStreamSynchronize(st));
    return MYPBR_OK;
}

constexpr size_t kWorkspaceMost = size_t(1) << 30;
struct Kept {
    std::mutex busy;
    char* p = nullptr;
    size_t bytes = 0;
};
Kept g_kept[kMaxDevices];

}  // namespace

int copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (bytes >= kSplitFrom)  // the parts are copied on streams of their own
        MYPBR_CUDA(cudaStreamSynchronize(st));
    return copy(dst, src, bytes, true, st);
}

int copy_to_device(void* dst, const void* src, size_t bytes) { return copy(dst, src, bytes, false, nullptr); }

int Workspace::reserve(size_t bytes) {
    int device = 0;
    MYPBR_CUDA(cudaGetDevice(&device));
    used_ = 0;
    if (bytes <= kWorkspaceMost && device < kMaxDevices && g_kept[device].busy.try_lock()) {
        Kept& k = g_kept[device];
        kept_ = device;
        if (k.bytes < bytes) {
            if (k.p)
                cudaFree(k.p);
            k.p = nullptr;
            k.bytes = 0;
            cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&k.p), bytes);
            if (e != cudaSuccess)
                return cuda_fail(e, "workspace");
            k.bytes = bytes;
        }
        base_ = k.p;
        return MYPBR_OK;
    }
    MYPBR_CUDA(cudaMalloc(reinterpret_cast<void**>(&base_), std::max<size_t>(bytes, 1)));
    return MYPBR_OK;
}

Workspace::~Workspace() {
    if (kept_ >= 0)
        g_kept[kept_].busy.unlock();
    else if (base_)
        cudaFree(base_);
}

void release_workspaces() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device >= kMaxDevices || !g_kept[device].busy.try_lock())
        return;
    Kept& k = g_kept[device];
    if (k.p)
        cudaFree(k.p);
    k.p = nullptr;
    k.bytes = 0;
    k.busy.unlock();
}

}  // namespace mypbr_dev
