// host_copy.cuh -- copies between device buffers and the caller's arrays.
//
// The caller's arrays are ordinary (pageable) Fortran or numpy memory as a rule.
// The driver copies such memory through a buffer of its own, one array after
// another with a wait each, at 3 to 8 GB/s.  Here the pieces of all arrays of a
// call go through page-locked chunks of the handle: the DMA of one chunk runs
// while the one before it is copied to (from) the caller's memory, by up to four
// threads from 4 MiB on.  Page-locked arrays (and managed or
// device ones) are copied directly.  Every call returns when its copies are complete.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <new>
#include <thread>
#include <vector>

namespace sph {

struct HostSeg {
    void* host;
    void* dev;
    size_t bytes;
    bool joined = false;      // the device range goes on where the segment before it ends
};

class HostCopy {
public:
    ~HostCopy() { release(); }
    void release() {
        for (int t = 0; t < kLanes; ++t) {
            for (int k = 0; k < 2; ++k)
                if (lane_[t].ev[k]) cudaEventDestroy(lane_[t].ev[k]);
        }
        if (first_ && registered_) {
            cudaHostUnregister(first_);
            free(first_);
        } else if (first_) {
            cudaFreeHost(first_);
        }
        if (rest_) cudaFreeHost(rest_);
        if (grown_) cudaFreeHost(grown_);
        first_ = rest_ = grown_ = nullptr;
        registered_ = false;
        chunk_ = kChunk;
        for (Lane& l : lane_) l = Lane{};
    }
    // The chunks for an owner whose usual copies are of `usual` bytes, with `extra`
    // zeroed bytes of page-locked memory behind the first lane's, which the caller may
    // use until release().
    //
    // A small owner takes small chunks, of ordinary memory that is page-locked
    // afterwards: to lock and unlock 0.25 / 0.5 / 1 MiB so takes 0.73 / 1.00 / 1.48 ms,
    // to allocate and free locked memory 1.6 to 2.8 ms whatever the size.  Its first
    // copy of more than both (a pair list) takes the full-size block: with the small
    // chunks those copies stayed 20 us (a tenth) slower.  A new
    // handle of 2,209 particles with its first upload and its end: 3.8 ms with a
    // full-size block, 1.4 ms.
    cudaError_t reserve(size_t usual, size_t extra, void** mem) {
        if (first_) return cudaErrorInvalidValue;
        const size_t c = (usual + kPage - 1) & ~(kPage - 1);
        const size_t bytes = (2 * std::max(c, kLeast) + extra + kPage - 1) & ~(kPage - 1);
        if (bytes <= kRegister) {
            void* p = aligned_alloc(kPage, bytes);
            if (p && cudaHostRegister(p, bytes, cudaHostRegisterMapped) == cudaSuccess) {
                first_ = p;
                registered_ = true;
                chunk_ = std::max(c, kLeast);
            } else {
                cudaGetLastError();
                free(p);               // (not to be had: a block of full-size chunks)
            }
        }
        const cudaError_t e = open_first(extra);
        if (e != cudaSuccess) return e;
        if (usual >= kShare) open_rest();
        *mem = (char*)first_ + 2 * chunk_;
        memset(*mem, 0, extra);
        return cudaSuccess;
    }
    // Device to host (to_host) or host to device on `stream`; complete on return.
    // Null host pointers are skipped.
    cudaError_t copy(int device, cudaStream_t stream, std::initializer_list<HostSeg> segs, bool to_host) {
        cudaError_t e;
        try {
            e = copy_segs(device, stream, segs, to_host);
        } catch (...) {
            e = cudaErrorMemoryAllocation;
        }
        // after a failure too: what was queued before it is at the caller's memory
        if (e != cudaSuccess) cudaStreamSynchronize(stream);
        return e;
    }

private:
    cudaError_t copy_segs(int device, cudaStream_t stream, std::initializer_list<HostSeg> segs, bool to_host) {
        std::vector<HostSeg> pageable, pieces;
        size_t total = 0;
        for (const HostSeg& s : segs) {
            if (!s.host || s.bytes == 0) continue;
            if (known(s.host)) {
                const cudaError_t e = cudaMemcpyAsync(to_host ? s.host : s.dev, to_host ? s.dev : s.host, s.bytes,
                                                      cudaMemcpyDefault, stream);
                if (e != cudaSuccess) return e;
                continue;
            }
            pageable.push_back(s);
            total += s.bytes;
        }
        int lanes = 1;
        if (total > 0) {
            const cudaError_t e = open(total, lanes);
            if (e != cudaSuccess) return e;
        }
        for (const HostSeg& s : pageable)
            for (size_t o = 0; o < s.bytes; o += chunk_)
                pieces.push_back({(char*)s.host + o, (char*)s.dev + o, std::min(s.bytes - o, chunk_),
                                  s.joined || o > 0});
        // small pieces share a chunk, and joined ones a DMA
        std::vector<Chunk> chunks;
        for (const HostSeg& p : pieces) {
            if (chunks.empty() || pad(chunks.back().bytes) + p.bytes > chunk_) chunks.push_back(Chunk{});
            Chunk& c = chunks.back();
            const bool next = p.joined && !c.dma.empty() && c.dma.back().dev + c.dma.back().bytes == p.dev;
            const size_t at = next ? c.bytes : pad(c.bytes);
            if (next) c.dma.back().bytes += p.bytes;
            else c.dma.push_back({(char*)p.dev, at, p.bytes});
            c.piece.push_back({(char*)p.host, at, p.bytes});
            c.bytes = at + p.bytes;
        }
        std::atomic<int> err{cudaSuccess};
        auto work = [&](int t) {
            if (t > 0) cudaSetDevice(device);
            const cudaError_t e = run_lane(lane_[t], stream, chunks, t, lanes, to_host);
            if (e != cudaSuccess) err = e;
        };
        std::thread helper[kLanes];
        int started = 1;
        for (; started < lanes; ++started) {
            try {
                helper[started] = std::thread(work, started);
            } catch (...) {
                break;       // no more threads (or no memory for one): this one takes their chunks
            }
        }
        work(0);
        for (int t = started; t < lanes; ++t) work(t);
        for (int t = 1; t < started; ++t) helper[t].join();
        const cudaError_t e = cudaStreamSynchronize(stream);
        return err != cudaSuccess ? (cudaError_t)err.load() : e;
    }

    // Chunk and lanes, us for 1.0 / 3.2 / 31 / 210 MB to the host, 16 cores: 1 lane with
    // chunks of 128 KiB 87 / 295 / 2760 / 21150, 256 KiB 71 / 241 / 2220 / 19320, 1 MiB
    // 74 / 228 / 1930 / 17210; with 1 MiB 2 lanes 84 / 182 / 1440 / 9150, 3 lanes
    // 93 / 165 / 1130 / 6980, 4 lanes 104 / 165 / 1270 / 5680, 6 lanes 140 / 179 / 1490 /
    // 5650, 8 lanes 183 / 194 / 1360 / 5840 (a thread costs about 10 us to start).
    // The other lanes would pay from 2 MB on, but their page-locked memory takes 4 to
    // 5.5 ms once: they begin at 4 MiB.  An owner whose usual copies are that large
    // gets it from reserve, not in its first copy.
    static constexpr size_t kChunk = size_t(1) << 20;      // 8 MiB held at most
    static constexpr size_t kShare = size_t(4) << 20;
    static constexpr int kLanes = 4;
    static constexpr size_t kPage = 4096, kLeast = size_t(64) << 10, kRegister = size_t(1) << 20;
    struct Part {
        char* host;
        size_t off, bytes;     // place in the chunk
    };
    struct Dma {
        char* dev;
        size_t off, bytes;
    };
    struct Chunk {
        std::vector<Part> piece;
        std::vector<Dma> dma;
        size_t bytes = 0;
    };
    struct Lane {
        void* buf[2] = {nullptr, nullptr};
        cudaEvent_t ev[2] = {nullptr, nullptr};
    };
    Lane lane_[kLanes];
    // Page-locked memory: one block for the first lane, one for the others, since an
    // allocation takes 1 to 2.8 ms up to 2 MiB.
    void* first_ = nullptr;
    void* rest_ = nullptr;
    void* grown_ = nullptr;        // a small owner's full-size chunks
    bool registered_ = false;      // first_ is ordinary memory, locked
    size_t chunk_ = kChunk;
    cudaError_t open_first(size_t extra) {
        return first_ ? cudaSuccess : cudaHostAlloc(&first_, 2 * chunk_ + extra, cudaHostAllocDefault);
    }
    void open_rest() {
        if (!rest_ && cudaHostAlloc(&rest_, (kLanes - 1) * 2 * chunk_, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            rest_ = nullptr;           // (one lane, then)
        }
    }
    // The lanes for a copy of `total` bytes.
    cudaError_t open(size_t total, int& lanes) {
        cudaError_t e = open_first(0);
        if (e != cudaSuccess) return e;
        if (chunk_ < kChunk && total > 2 * chunk_) {
            if (cudaHostAlloc(&grown_, 2 * kChunk, cudaHostAllocDefault) == cudaSuccess) {
                chunk_ = kChunk;
            } else {
                cudaGetLastError();
                grown_ = nullptr;      // (the small ones, then)
            }
        }
        if (total >= kShare) {
            open_rest();
            const unsigned hw = std::thread::hardware_concurrency();
            if (rest_) lanes = hw >= 8 ? kLanes : hw >= 4 ? 2 : 1;
        }
        for (int t = 0; t < lanes; ++t)
            for (int k = 0; k < 2; ++k) {
                lane_[t].buf[k] = t == 0 ? (char*)(grown_ ? grown_ : first_) + k * chunk_ : (char*)rest_ + (2 * (t - 1) + k) * chunk_;
                if (!lane_[t].ev[k] &&
                    (e = cudaEventCreateWithFlags(&lane_[t].ev[k], cudaEventDisableTiming)) != cudaSuccess)
                    return e;
            }
        return e;
    }

    static size_t pad(size_t b) { return (b + 255) & ~size_t(255); }
    // Page-locked, managed or device memory: the runtime can copy it directly, and
    // device memory is not the CPU's to touch.
    static bool known(const void* p) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
        return a.type != cudaMemoryTypeUnregistered;
    }
    // Chunks t, t + lanes, ...: two buffers, the DMA of one while the other is
    // copied by this thread.
    static cudaError_t run_lane(Lane& l, cudaStream_t stream, const std::vector<Chunk>& chunks, int t, int lanes,
                                bool to_host) {
        cudaError_t e = cudaSuccess;
        const Chunk* behind = nullptr;          // to host: the chunk whose DMA is in flight
        int k = 0;
        auto unpack = [&](const Chunk& c, int b) {
            if ((e = cudaEventSynchronize(l.ev[b])) != cudaSuccess) return;
            for (const Part& q : c.piece) memcpy(q.host, (char*)l.buf[b] + q.off, q.bytes);
        };
        bool used[2] = {false, false};
        for (size_t i = t; i < chunks.size() && e == cudaSuccess; i += lanes, k ^= 1) {
            const Chunk& c = chunks[i];
            if (!to_host && used[k]) e = cudaEventSynchronize(l.ev[k]);      // its DMA must be done
            char* pin = (char*)l.buf[k];
            if (!to_host && e == cudaSuccess)
                for (const Part& q : c.piece) memcpy(pin + q.off, q.host, q.bytes);
            for (const Dma& d : c.dma) {
                if (e != cudaSuccess) break;
                e = to_host ? cudaMemcpyAsync(pin + d.off, d.dev, d.bytes, cudaMemcpyDeviceToHost, stream)
                            : cudaMemcpyAsync(d.dev, pin + d.off, d.bytes, cudaMemcpyHostToDevice, stream);
            }
            if (e == cudaSuccess) e = cudaEventRecord(l.ev[k], stream);
            used[k] = true;
            if (to_host && behind && e == cudaSuccess) unpack(*behind, k ^ 1);
            behind = &c;
        }
        if (to_host && behind && e == cudaSuccess) unpack(*behind, k ^ 1);
        return e;
    }
};

}  // namespace sph
