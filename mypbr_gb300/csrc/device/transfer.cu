// See transfer.h.
#include "transfer.h"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <thread>
#include <vector>

#include "cuda_check.h"

namespace mypbr_dev {
namespace {

constexpr int kMaxDevices = 64;

// The GPU reads and writes pageable host memory through the host's page
// tables, at its full rate wherever the pages exist (50 MiB in 0.31 ms and out
// in 0.28; through pinned buffers and eight threads 0.84 and 0.93 ms). Pages
// of a frame that the caller has just allocated do not, and each costs about
// 50 us when the transfer is the first to meet it (9.8 MB, 150 pages of 64
// KiB: 7.5 ms), but 2 us when the host writes to it first (0.31 ms, and 0.09
// for the transfer). Four threads make 50 MiB of pages in half the time of
// one (1.26 ms); starting them takes about 0.1 ms, a third of what 9.8 MB take.
constexpr size_t kMakeFrom = size_t(64) << 10;
constexpr int kThreads = 4;
constexpr size_t kThreadsFrom = size_t(16) << 20;

// Whether p is pageable host memory. Registered and managed memory has its
// pages, and a device pointer is the driver's to refuse.
bool pageable(const void* p) {
    cudaPointerAttributes a = {};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// How many of the pages of [p, p + bytes) do not exist; make: writes a byte of
// the frame in each of them. (A plain store: one that reads first would get
// the zero page and take a second fault, 25 us.)
size_t missing_pages(char* p, size_t bytes, size_t page, bool make) {
    char* const end = p + bytes;
    char* at = p - reinterpret_cast<uintptr_t>(p) % page;
    unsigned char there[4096];
    size_t missing = 0;
    while (at < end) {
        const size_t pages = std::min(sizeof there, (size_t(end - at) + page - 1) / page);
        if (mincore(at, pages * page, there) != 0)
            return 0;
        for (size_t k = 0; k < pages; k++, at += page)
            if (!(there[k] & 1)) {
                missing++;
                if (make)
                    *static_cast<volatile char*>(std::max(at, p)) = 0;
            }
    }
    return missing;
}

// Makes the pages of memory that is about to be written.
void make_pages(char* p, size_t bytes) {
    const size_t page = size_t(sysconf(_SC_PAGESIZE));
    if (missing_pages(p, bytes, page, false) * page < kThreadsFrom) {
        missing_pages(p, bytes, page, true);
        return;
    }
    const size_t part = (bytes / kThreads / page + 1) * page;
    auto run = [=](int t) {
        const size_t at = std::min(bytes, part * size_t(t));
        missing_pages(p + at, std::min(part, bytes - at), page, true);
    };
    std::thread pool[kThreads];
    try {
        for (int t = 1; t < kThreads; t++)
            pool[t] = std::thread(run, t);
    } catch (...) {  // no more threads to be had: the transfer makes the other pages
    }
    run(0);
    for (std::thread& t : pool)
        if (t.joinable())
            t.join();
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
    if (bytes >= kMakeFrom && pageable(dst))
        make_pages(static_cast<char*>(dst), bytes);
    MYPBR_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    MYPBR_CUDA(cudaStreamSynchronize(st));
    return MYPBR_OK;
}

int copy_to_device(void* dst, const void* src, size_t bytes) {
    MYPBR_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
    return MYPBR_OK;
}

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
            if (e != cudaSuccess) {
                cudaGetLastError();
                return cuda_fail(e, "workspace");
            }
            k.bytes = bytes;
        }
        base_ = k.p;
        return MYPBR_OK;
    }
    MYPBR_CUDA(device_malloc(&base_, std::max<size_t>(bytes, 1)));
    return MYPBR_OK;
}

Workspace::~Workspace() {
    if (kept_ >= 0)
        g_kept[kept_].busy.unlock();
    else if (base_)
        cudaFree(base_);
}

cudaError_t device_malloc_bytes(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        release_workspaces();
        e = cudaMalloc(p, bytes);
        cudaGetLastError();  // or the next check of a launch would report it
    }
    return e;
}

namespace {
constexpr size_t kWordsInBlock = 16384;
struct HostWords {
    std::mutex busy;
    std::vector<int*> blocks, left;  // `left` has room for every word there is
};
// Never destroyed: a program's last handles may go after this library's objects.
HostWords& host_words() {
    static HostWords* const words = new HostWords;
    return *words;
}
}  // namespace

int* take_host_word() {
    HostWords& w = host_words();
    std::lock_guard<std::mutex> lock(w.busy);
    if (w.left.empty()) {
        int* block = nullptr;
        try {
            w.blocks.reserve(w.blocks.size() + 1);
            w.left.reserve((w.blocks.size() + 1) * kWordsInBlock);
        } catch (...) {
            return nullptr;
        }
        if (cudaHostAlloc(reinterpret_cast<void**>(&block), kWordsInBlock * sizeof(int),
                          cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        w.blocks.push_back(block);
        for (size_t k = kWordsInBlock; k-- > 0;)
            w.left.push_back(block + k);
    }
    int* const word = w.left.back();
    w.left.pop_back();
    *word = 0;
    return word;
}

void give_host_word(int* word) {
    if (!word)
        return;
    HostWords& w = host_words();
    std::lock_guard<std::mutex> lock(w.busy);
    w.left.push_back(word);
}

namespace {
// once no word is taken
void release_host_words() {
    HostWords& w = host_words();
    std::lock_guard<std::mutex> lock(w.busy);
    if (w.left.size() != w.blocks.size() * kWordsInBlock)
        return;
    for (int* block : w.blocks)
        cudaFreeHost(block);
    w.blocks.clear();
    w.left.clear();
}

// unless a call uses it
void release(Kept& k) {
    if (!k.busy.try_lock())
        return;
    if (k.p)
        cudaFree(k.p);
    k.p = nullptr;
    k.bytes = 0;
    k.busy.unlock();
}
}  // namespace

void release_workspaces() {
    int device = 0;
    if (cudaGetDevice(&device) == cudaSuccess && device < kMaxDevices)
        release(g_kept[device]);
}

}  // namespace mypbr_dev

extern "C" int mypbr_gpu_release_memory(void) {
    for (mypbr_dev::Kept& k : mypbr_dev::g_kept)
        mypbr_dev::release(k);
    mypbr_dev::release_host_words();
    return MYPBR_OK;
}
