// host_copy.cuh -- copies between device buffers and the caller's arrays.
//
// The caller's arrays are ordinary (pageable) Fortran or numpy memory as a rule.
// The driver copies such memory through a buffer of its own, one array after
// another with a wait each, at 3 to 8 GB/s.  Here the pieces of all arrays of a
// call go through page-locked chunks of the handle: the DMA of one chunk runs
// while the one before it is copied to (from) the caller's memory, by up to four
// threads when there is enough to share.  Page-locked arrays (and managed or
// device ones) are copied directly.  Every call returns when its copies are complete.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
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
        for (void** b : {&first_, &rest_}) {
            if (*b) cudaFreeHost(*b);
            *b = nullptr;
        }
        for (Lane& l : lane_) l = Lane{};
    }
    // The first lane's chunks with `extra` zeroed bytes of page-locked memory behind
    // them, which the caller may use until release().
    cudaError_t reserve(size_t extra, void** mem) {
        const cudaError_t e = open(1, extra);
        if (e != cudaSuccess) return e;
        *mem = (char*)first_ + 2 * kChunk;
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
        std::vector<HostSeg> pieces;
        size_t total = 0;
        for (const HostSeg& s : segs) {
            if (!s.host || s.bytes == 0) continue;
            if (known(s.host)) {
                const cudaError_t e = cudaMemcpyAsync(to_host ? s.host : s.dev, to_host ? s.dev : s.host, s.bytes,
                                                      cudaMemcpyDefault, stream);
                if (e != cudaSuccess) return e;
                continue;
            }
            for (size_t o = 0; o < s.bytes; o += kChunk)
                pieces.push_back({(char*)s.host + o, (char*)s.dev + o, s.bytes - o < kChunk ? s.bytes - o : kChunk,
                                  s.joined || o > 0});
            total += s.bytes;
        }
        // small pieces share a chunk, and joined ones a DMA
        std::vector<Chunk> chunks;
        for (const HostSeg& p : pieces) {
            if (chunks.empty() || pad(chunks.back().bytes) + p.bytes > kChunk) chunks.push_back(Chunk{});
            Chunk& c = chunks.back();
            const bool next = p.joined && !c.dma.empty() && c.dma.back().dev + c.dma.back().bytes == p.dev;
            const size_t at = next ? c.bytes : pad(c.bytes);
            if (next) c.dma.back().bytes += p.bytes;
            else c.dma.push_back({(char*)p.dev, at, p.bytes});
            c.piece.push_back({(char*)p.host, at, p.bytes});
            c.bytes = at + p.bytes;
        }
        int lanes = 1;
        if (total >= kShare) {
            const unsigned hw = std::thread::hardware_concurrency();
            lanes = hw >= 8 ? kLanes : hw >= 4 ? 2 : 1;
        }
        if (!chunks.empty()) {
            const cudaError_t e = open(lanes, 0);
            if (e != cudaSuccess) return e;
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

    static constexpr size_t kChunk = size_t(1) << 20;      // 1 MiB: 20 us of PCIe, 8 MiB held at most
    static constexpr size_t kShare = size_t(4) << 20;      // a thread costs about 30 us to start
    static constexpr int kLanes = 4;
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
    // Page-locked memory: one allocation for the first lane, one for the others, since
    // each takes 0.8 to 2.6 ms whatever its size.
    void* first_ = nullptr;
    void* rest_ = nullptr;
    cudaError_t open(int lanes, size_t extra) {
        cudaError_t e = cudaSuccess;
        if (!first_ && (e = cudaHostAlloc(&first_, 2 * kChunk + extra, cudaHostAllocDefault)) != cudaSuccess) return e;
        if (lanes > 1 && !rest_ &&
            (e = cudaHostAlloc(&rest_, (kLanes - 1) * 2 * kChunk, cudaHostAllocDefault)) != cudaSuccess)
            return e;
        for (int t = 0; t < lanes; ++t)
            for (int k = 0; k < 2; ++k) {
                lane_[t].buf[k] = t == 0 ? (char*)first_ + k * kChunk : (char*)rest_ + (2 * (t - 1) + k) * kChunk;
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
