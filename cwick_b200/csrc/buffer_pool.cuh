// buffer_pool.cuh -- device buffers that go from one context to the next.
//
// A context that goes leaves its work buffers to the next one on its device: a server makes and drops contexts with its
// request slots, and a few megabytes from cudaMalloc take half a millisecond of the next slot's first call. At most
// POOL_BYTES per device wait here; they are given back when the device's last context goes, or when an allocation fails.
//
// What comes in has no user left, by the caller's word (`idle`): it knows every stream on which the buffer was used and has
// waited for them. A buffer of which that is not known is freed, and cudaFree waits for whatever is still in flight.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

// Where a context's buffers are in use. Known while all its work goes to one stream; work captured into a graph runs where
// the graph is launched, and a stream that the context had before may still have work: from then on it is not known.
class CwkBufferUse {
public:
    // With every use of a buffer: `stream` is the context's.
    void use(cudaStream_t stream) {
        if (!known_) return;
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) (void)cudaGetLastError();
        else if (st != cudaStreamCaptureStatusNone) known_ = false;
    }
    void lose() { known_ = false; }
    bool known() const { return known_; }
    // Waits until no work is left that uses the buffers, where that is known. No device-wide wait: while another thread's stream is in
    // capture it is refused, and spoils the capture. Nor is a stream waited for that is itself part of a capture, which the
    // legacy stream is as soon as any blocking stream is.
    bool idle(cudaStream_t stream) const {
        if (!known_) return false;
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone && cudaStreamSynchronize(stream) == cudaSuccess) return true;
        (void)cudaGetLastError();
        return false;
    }

private:
    bool known_ = true;
};

class CwkBufferPool {
public:
    static constexpr size_t POOL_BYTES = 384u << 20;      // one of the largest workspaces (gdn_chunk.cu, 320 MB), or many of the others

    void add_context(int device) {
        std::lock_guard<std::mutex> l(mu_);
        pools_[device].contexts++;
    }
    // The device is current. The last context's going gives the buffers back.
    void drop_context(int device) {
        std::vector<Buffer> last;
        {
            std::lock_guard<std::mutex> l(mu_);
            Pool &pool = pools_[device];
            if (--pool.contexts == 0) last = take_all(pool);
        }
        for (const Buffer &b : last) cudaFree(b.p);
    }
    // At least `bytes` on the current device, which is `device`; *granted is what there is. On an error neither is written.
    cudaError_t alloc(int device, size_t bytes, void **p, size_t *granted) {
        std::vector<Buffer> waiting;
        {
            std::lock_guard<std::mutex> l(mu_);
            Pool &pool = pools_[device];
            int best = -1;
            for (int i = 0; i < (int)pool.waiting.size(); i++) {
                const size_t have = pool.waiting[i].bytes;
                if (have >= bytes && have / 4 <= bytes && (best < 0 || have < pool.waiting[best].bytes)) best = i;
            }
            if (best >= 0) {
                *p = pool.waiting[best].p;
                *granted = pool.waiting[best].bytes;
                pool.held -= *granted;
                pool.waiting.erase(pool.waiting.begin() + best);
                return cudaSuccess;
            }
        }
        void *d = nullptr;
        cudaError_t e = cudaMalloc(&d, bytes);
        if (e == cudaErrorMemoryAllocation) {              // what waits here may be what is missing
            {
                std::lock_guard<std::mutex> l(mu_);
                waiting = take_all(pools_[device]);
            }
            if (!waiting.empty()) {
                (void)cudaGetLastError();
                for (const Buffer &b : waiting) cudaFree(b.p);
                e = cudaMalloc(&d, bytes);
            }
        }
        if (e != cudaSuccess) return e;
        *p = d;
        *granted = bytes;
        return cudaSuccess;
    }
    cudaError_t free(int device, void *p, size_t bytes, bool idle) {
        if (!p) return cudaSuccess;
        if (idle) {
            std::lock_guard<std::mutex> l(mu_);
            Pool &pool = pools_[device];
            if (pool.contexts > 0 && pool.held + bytes <= POOL_BYTES) {
                pool.waiting.push_back({p, bytes});
                pool.held += bytes;
                return cudaSuccess;
            }
        }
        return cudaFree(p);
    }

private:
    struct Buffer {
        void *p;
        size_t bytes;
    };
    struct Pool {
        std::vector<Buffer> waiting;
        size_t held = 0;
        int contexts = 0;
    };
    static std::vector<Buffer> take_all(Pool &pool) {
        std::vector<Buffer> all;
        all.swap(pool.waiting);
        pool.held = 0;
        return all;
    }
    std::mutex mu_;
    std::map<int, Pool> pools_;
};
