// The frame copies (csrc/device/transfer.cu) against a CUDA runtime made of
// host memory, for what no GPU is needed to see: which calls they make, in
// which order, and what they do when one fails. One scenario per run, named
// on the command line; exit code 0 when it holds.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "../mypbr_gb300/csrc/device/transfer.cu"

namespace {

struct Fake {
    size_t left = SIZE_MAX;      // device memory, bytes
    std::map<void*, size_t> held;
    int copies = 0, pinned = 0;  // transfers; pinned blocks
    size_t pinned_left = SIZE_MAX;
    bool pages_made = false;     // when the transfer started
    const char* host = nullptr;  // the caller's memory and what the driver calls it
    cudaMemoryType kind = cudaMemoryTypeUnregistered;
} fake;

}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > fake.left)
        return cudaErrorMemoryAllocation;
    fake.left -= n;
    *p = std::malloc(n);
    fake.held[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    fake.left += fake.held[p];
    fake.held.erase(p);
    return std::free(p), cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (n > fake.pinned_left)
        return cudaErrorMemoryAllocation;
    fake.pinned++;
    return *p = std::malloc(n), cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    fake.pinned--;
    return std::free(p), cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = p == fake.host ? fake.kind : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    fake.copies++;
    if ((d == fake.host || s == fake.host) && fake.kind == cudaMemoryTypeDevice)
        return cudaErrorInvalidValue;
    fake.pages_made = mypbr_dev::missing_pages(static_cast<char*>(d), n, size_t(sysconf(_SC_PAGESIZE)), false) == 0;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
}

int mypbr_dev::cuda_fail(cudaError_t e, const char*) {
    return e == cudaErrorMemoryAllocation ? MYPBR_ERR_OUT_OF_MEMORY : MYPBR_ERR_CUDA;
}

namespace {

#define HOLDS(x)                                              \
    do {                                                      \
        if (!(x)) {                                           \
            std::fprintf(stderr, "does not hold: %s\n", #x);  \
            std::exit(1);                                     \
        }                                                     \
    } while (0)

constexpr size_t kBytes = (size_t(20) << 20) + 24;

std::vector<char> pattern() {
    std::vector<char> v(kBytes);
    for (size_t k = 0; k < kBytes; k++)
        v[k] = char(k * 7 + k / 4096);
    return v;
}

// Each way one transfer, whatever kind of host memory it is.
void one_transfer(cudaMemoryType kind) {
    std::vector<char> a = pattern(), dev(kBytes), back(kBytes);
    fake.kind = kind;
    fake.host = a.data();
    HOLDS(mypbr_dev::copy_to_device(dev.data(), a.data(), kBytes) == MYPBR_OK && fake.copies == 1);
    fake.host = back.data();
    HOLDS(mypbr_dev::copy_to_host(back.data(), dev.data(), kBytes, nullptr) == MYPBR_OK && fake.copies == 2);
    HOLDS(back == a);
}

// A new frame's pages exist when its transfer starts, and nothing around it is written; pages that exist keep their contents.
void pages_are_made(size_t bytes, size_t offset) {
    const size_t page = size_t(sysconf(_SC_PAGESIZE)), size = (offset + bytes + 2 * page) / page * page;
    char* const map = static_cast<char*>(mmap(nullptr, size, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    HOLDS(map != MAP_FAILED);
    std::vector<char> a(bytes, 3);
    HOLDS(mypbr_dev::copy_to_host(map + offset, a.data(), bytes, nullptr) == MYPBR_OK);
    HOLDS(fake.pages_made && std::memcmp(map + offset, a.data(), bytes) == 0);
    mypbr_dev::make_pages(map + offset, bytes);
    HOLDS(std::memcmp(map + offset, a.data(), bytes) == 0);
    unsigned char there = 0;  // the page after the frame's last one
    HOLDS(mincore(map + (offset + bytes + page - 1) / page * page, page, &there) == 0 && !(there & 1));
    munmap(map, size);
}

// A device pointer where host memory is asked for: nothing here may touch it.
void device_pointers_are_refused() {
    std::vector<char> dev(kBytes);
    char* const bad = reinterpret_cast<char*>(0x1000);
    fake.kind = cudaMemoryTypeDevice;
    fake.host = bad;
    HOLDS(mypbr_dev::copy_to_device(dev.data(), bad, kBytes) == MYPBR_ERR_CUDA);
    HOLDS(mypbr_dev::copy_to_host(bad, dev.data(), kBytes, nullptr) == MYPBR_ERR_CUDA);
}

// Memory that the kept workspace holds between calls is there for any allocation, and stays while a call uses it.
void kept_memory_is_given_back() {
    constexpr size_t MiB = size_t(1) << 20;
    fake.left = 4 * MiB;
    void* p = nullptr;
    {
        mypbr_dev::Workspace w;
        HOLDS(w.reserve(3 * MiB) == MYPBR_OK);
        HOLDS(mypbr_dev::device_malloc(&p, 2 * MiB) == cudaErrorMemoryAllocation && fake.left == 1 * MiB);
        mypbr_dev::Workspace other;  // as a second thread's call: memory of its own
        HOLDS(other.reserve(2 * MiB) == MYPBR_ERR_OUT_OF_MEMORY);
        HOLDS(other.reserve(1 * MiB) == MYPBR_OK);
    }
    HOLDS(fake.left == 1 * MiB);
    HOLDS(mypbr_dev::device_malloc(&p, 2 * MiB) == cudaSuccess && fake.left == 2 * MiB);
    HOLDS(mypbr_dev::device_malloc(&p, 3 * MiB) == cudaErrorMemoryAllocation);
}

// The public call gives back what no call is using.
void released_on_request() {
    fake.left = 1000;
    {
        mypbr_dev::Workspace w;
        HOLDS(w.reserve(600) == MYPBR_OK);
        HOLDS(mypbr_gpu_release_memory() == MYPBR_OK && fake.left == 400);
    }
    HOLDS(fake.left == 400);
    HOLDS(mypbr_gpu_release_memory() == MYPBR_OK && fake.left == 1000);
    HOLDS(mypbr_gpu_release_memory() == MYPBR_OK && fake.left == 1000);
}

// Words of several blocks: each its own, zero when taken, the blocks freed on request once none is taken.
void host_words() {
    std::vector<int*> taken;
    std::set<int*> different;
    for (int k = 0; k < 40000; k++) {
        taken.push_back(mypbr_dev::take_host_word());
        HOLDS(taken.back() && *taken.back() == 0);
        *taken.back() = k + 1;
        different.insert(taken.back());
    }
    HOLDS(different.size() == taken.size() && fake.pinned == 3);
    fake.pinned_left = 0;
    while (int* word = mypbr_dev::take_host_word())
        taken.push_back(word);
    HOLDS(taken.size() == 3 * 16384);
    mypbr_dev::give_host_word(taken.back());
    taken.pop_back();
    HOLDS(mypbr_gpu_release_memory() == MYPBR_OK && fake.pinned == 3);
    for (int* word : taken)
        mypbr_dev::give_host_word(word);
    mypbr_dev::give_host_word(nullptr);
    HOLDS(mypbr_gpu_release_memory() == MYPBR_OK && fake.pinned == 0);
    HOLDS(!mypbr_dev::take_host_word());
    fake.pinned_left = SIZE_MAX;
    HOLDS(mypbr_dev::take_host_word() && fake.pinned == 1);
}

// More than is ever kept: the kept workspace makes room for it, and it is given back at once.
void large_workspaces_are_not_kept() {
    constexpr size_t GiB = size_t(1) << 30;
    fake.left = 2 * GiB;
    {
        mypbr_dev::Workspace w;
        HOLDS(w.reserve(GiB) == MYPBR_OK);
    }
    {
        mypbr_dev::Workspace w;
        HOLDS(w.reserve(GiB + GiB / 2) == MYPBR_OK && fake.left == GiB / 2);
    }
    HOLDS(fake.left == 2 * GiB);
}

}  // namespace

int main(int argc, char** argv) {
    const std::string name = argc > 1 ? argv[1] : "";
    if (name == "pageable")
        one_transfer(cudaMemoryTypeUnregistered);
    else if (name == "pinned")
        one_transfer(cudaMemoryTypeHost);
    else if (name == "managed")
        one_transfer(cudaMemoryTypeManaged);
    else if (name == "device")
        device_pointers_are_refused();
    else if (name == "new_frame")  // <bytes> <offset in the mapping>
        pages_are_made(std::strtoull(argv[2], nullptr, 10), std::strtoull(argv[3], nullptr, 10));
    else if (name == "out_of_memory")
        kept_memory_is_given_back();
    else if (name == "release")
        released_on_request();
    else if (name == "words")
        host_words();
    else if (name == "large")
        large_workspaces_are_not_kept();
    else
        return 2;
    return 0;
}
