// host_copy.cuh over a CUDA runtime of this file's own: copies are queued and done when
// their stream or event is waited for, "device" pointers are memory the CPU may not
// touch, and calls and allocations can be made to fail.  Prints what went wrong and
// exits 1.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <functional>
#include <mutex>
#include <set>
#include <vector>

#include "../sph-2d_b200/csrc/host_copy.cuh"

namespace {
std::recursive_mutex mu;
std::vector<std::function<void()>> queue;      // work queued and not yet done
size_t done = 0;                               // items of the queue that ran
std::set<const void*> locked, device;          // page-locked and device arrays (start address)
int memcpys, fail_memcpy = -1, fail_alloc = -1, allocs, registers;
long news, fail_new = -1;
bool armed = false;                            // operator new counts and may fail
thread_local bool inside = false;              // (not in this file's own calls)
cudaMemcpyKind last_kind[64];

void run_to(size_t n) {
    std::lock_guard<std::recursive_mutex> l(mu);
    for (; done < n; ++done) queue[done]();
}
size_t pending() { return queue.size() - done; }
}  // namespace

void* operator new(size_t n) {
    if (armed && !inside && __atomic_fetch_add(&news, 1, __ATOMIC_RELAXED) == fail_new) throw std::bad_alloc();
    void* p = malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

extern "C" {
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (memcpys < 64) last_kind[memcpys] = kind;
    if (memcpys++ == fail_memcpy) return cudaErrorInvalidValue;
    inside = true;
    // a "device" array that the CPU may not touch: nothing to move
    if (device.count(dst) || device.count(src)) queue.push_back([] {});
    else queue.push_back([=] { memcpy(dst, src, n); });
    inside = false;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { run_to(queue.size()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t) new size_t(0); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (size_t*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> l(mu);
    *(size_t*)e = queue.size();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { run_to(*(size_t*)e); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (allocs++ == fail_alloc) return cudaErrorMemoryAllocation;
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned) { ++registers; return allocs == fail_alloc ? cudaErrorMemoryAllocation : cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = locked.count(p) ? cudaMemoryTypeHost : device.count(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
}

namespace {
int bad = 0;
void expect(bool ok, const char* what, long k) {
    if (!ok) { printf("FAILED: %s (%ld)\n", what, k); bad = 1; }
}
void reset() {
    run_to(queue.size());
    queue.clear();
    done = 0;
    memcpys = allocs = registers = 0;
    fail_memcpy = fail_alloc = -1;
    news = 0;
    fail_new = -1;
    armed = false;
}
std::vector<char> filled(size_t n, char c) {
    std::vector<char> v(n);
    for (size_t i = 0; i < n; ++i) v[i] = (char)(c + i * 7);
    return v;
}
}  // namespace

int main(int argc, char** argv) {
    const bool only_device = argc > 1 && argv[1][0] == 'd';
    const size_t big = size_t(9) << 20, small = 100000;
    std::vector<char> dev_a(small), dev_b(big), want_a = filled(small, 1), want_b = filled(big, 2);
    std::vector<char> host_a(small), host_b(big);
    locked.insert(host_a.data());
    cudaStream_t st = (cudaStream_t)1;
    for (int dir = 0; dir < 2 && argc == 1; ++dir) {
        const bool to_host = dir == 1;
        std::vector<char>&src_a = to_host ? dev_a : host_a, &src_b = to_host ? dev_b : host_b;
        std::vector<char>&dst_a = to_host ? host_a : dev_a, &dst_b = to_host ? host_b : dev_b;
        auto call = [&](sph::HostCopy& c) {
            src_a = want_a; src_b = want_b;
            memset(dst_a.data(), 0, small); memset(dst_b.data(), 0, big);
            // a page-locked array first: its copy is queued before the rest can fail
            return c.copy(0, st, {{host_a.data(), dev_a.data(), small}, {host_b.data(), dev_b.data(), big}}, to_host);
        };
        auto right = [&] { return dst_a == want_a && dst_b == want_b; };
        {
            sph::HostCopy c;
            expect(call(c) == cudaSuccess && right() && pending() == 0, "plain copy", dir);
        }
        for (int k = 0; k < 48; ++k) {          // the k / 2-th copy fails, in a first call and in a later one
            reset();
            sph::HostCopy c;
            if (k & 1) call(c);
            reset();
            fail_memcpy = k / 2;
            const cudaError_t e = call(c);
            expect(e != cudaSuccess || right(), "copy failure", k);
            expect(pending() == 0, "copies in flight after a copy failed", k);
        }
        for (int k = 0; k < 3; ++k) {           // a small owner's larger blocks are refused
            reset();
            sph::HostCopy c;
            void* mem;
            c.reserve(1000, 64, &mem);
            fail_alloc = k;
            const cudaError_t e = call(c);
            expect(e == cudaSuccess && right() && pending() == 0, "refused block of a small owner", k);
        }
        for (int k = 0; k < 4; ++k) {           // page-locked memory is refused
            reset();
            sph::HostCopy c;
            if (k & 1) call(c);
            reset();
            fail_alloc = k / 2;
            const cudaError_t e = call(c);
            expect(e != cudaSuccess || right(), "allocation failure", k);
            expect(pending() == 0, "copies in flight after an allocation failed", k);
        }
        for (long k = 0; k < 80; ++k) {         // the k-th operator new fails (vectors, threads)
            reset();
            sph::HostCopy c;
            call(c);
            reset();
            src_a = want_a; src_b = want_b;
            memset(dst_a.data(), 0, small); memset(dst_b.data(), 0, big);
            fail_new = k;
            armed = true;
            const cudaError_t e = c.copy(0, st, {{host_a.data(), dev_a.data(), small}, {host_b.data(), dev_b.data(), big}}, to_host);
            armed = false;
            expect(e != cudaSuccess || right(), "no memory", k);
            expect(pending() == 0, "copies in flight without memory", k);
        }
    }
    if (argc > 1 && argv[1][0] == 'r') {
        // what a new owner takes, and that its copies are right with it
        for (size_t usual : {size_t(1000), size_t(130000), size_t(400000), size_t(600000), size_t(10) << 20}) {
            for (int refuse = 0; refuse < 2; ++refuse) {
                reset();
                sph::HostCopy c;
                void* mem = nullptr;
                fail_alloc = refuse ? 0 : -1;
                const bool small_owner = usual <= 500000;
                const cudaError_t e = c.reserve(usual, 200, &mem);
                expect(registers == (small_owner ? 1 : 0), "blocks of ordinary memory locked", (long)usual);
                const bool large_owner = usual >= (size_t(4) << 20);
                expect(allocs == (small_owner && !refuse ? 0 : large_owner && !refuse ? 2 : 1), "blocks of locked memory",
                       (long)usual);
                fail_alloc = -1;
                if (refuse) {
                    expect(e != cudaSuccess, "refused memory", (long)usual);
                    continue;
                }
                expect(e == cudaSuccess && mem, "reserve", (long)usual);
                for (int k = 0; k < 200; ++k) expect(((char*)mem)[k] == 0, "zeroed", k);
                memset(mem, 0x5a, 200);
                const int before = allocs;
                for (int n = 0; n < 3; ++n) {
                    for (size_t m : {size_t(1), size_t(4096), size_t(131073), size_t(700001), big}) {
                        for (int dir = 0; dir < 2; ++dir) {
                            std::vector<char>&src = dir ? dev_b : host_b, &dst = dir ? host_b : dev_b;
                            src = want_b;
                            memset(dst.data(), 0, big);
                            expect(c.copy(0, st, {{host_b.data(), dev_b.data(), m}}, dir == 1) == cudaSuccess, "copy", (long)m);
                            expect(!memcmp(dst.data(), want_b.data(), m) && (m == big || dst[m] == 0), "bytes", (long)m);
                        }
                    }
                }
                expect(allocs == before + (large_owner ? 0 : small_owner ? 2 : 1), "the large copies' blocks", (long)usual);
                for (int k = 0; k < 200; ++k) expect(((char*)mem)[k] == 0x5a, "the owner's memory", k);
            }
        }
        if (!bad) printf("ok\n");
        return bad;
    }
    if (only_device) {
        // the caller's array is on the device: the runtime copies it, the CPU does not touch it
        for (int dir = 0; dir < 2; ++dir) {
            reset();
            void* fence = mmap(nullptr, small, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            device.insert(fence);
            sph::HostCopy c;
            expect(c.copy(0, st, {{fence, dev_a.data(), small}}, dir == 1) == cudaSuccess, "device array", dir);
            expect(memcpys == 1 && last_kind[0] == cudaMemcpyDefault, "kind of the device array's copy", dir);
            expect(pending() == 0, "device array's copy in flight", dir);
        }
    }
    if (!bad) printf("ok\n");
    return bad;
}
