// The pool of device buffers (csrc/buffer_pool.cuh) against a fake of the CUDA calls that it makes.
#include "../../cwick_b200/csrc/buffer_pool.cuh"

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>

static std::mutex fake_mu;
static std::set<void *> live;
static size_t in_use, memory = SIZE_MAX;
static std::map<void *, size_t> size_of;
static int frees, syncs;
static bool sync_fails, query_fails;
static cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::mutex> l(fake_mu);
    if (in_use + n > memory) return cudaErrorMemoryAllocation;
    *p = malloc(1);
    live.insert(*p);
    size_of[*p] = n;
    in_use += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> l(fake_mu);
    if (!live.erase(p)) abort();
    in_use -= size_of[p];
    frees++;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { syncs++; return sync_fails ? cudaErrorUnknown : cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    if (query_fails) return cudaErrorStreamCaptureImplicit;
    *st = capture;
    return cudaSuccess;
}
}

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
constexpr size_t MB = 1u << 20;

int main() {
    const cudaStream_t stream = (cudaStream_t)1;
    {   // an idle buffer goes to the next context of its device, and to no other device's
        CwkBufferPool pool;
        void *a = nullptr, *b = nullptr;
        size_t na = 0, nb = 0;
        pool.add_context(0); pool.add_context(0); pool.add_context(16);
        CHECK(pool.alloc(0, 8 * MB, &a, &na) == cudaSuccess && na == 8 * MB);
        pool.free(0, a, na, true);
        CHECK(frees == 0);
        CHECK(pool.alloc(16, 8 * MB, &b, &nb) == cudaSuccess && b != a);
        pool.free(16, b, nb, true);
        CHECK(pool.alloc(0, 4 * MB, &b, &nb) == cudaSuccess && b == a && nb == 8 * MB);
        pool.free(0, b, nb, true);
        CHECK(pool.alloc(0, 1 * MB, &b, &nb) == cudaSuccess && b != a);      // more than four times what is asked for stays
        pool.free(0, b, nb, true);
        pool.drop_context(0);
        CHECK(frees == 0);
        pool.drop_context(0);
        CHECK(frees == 2);                                                   // the device's last context
        pool.drop_context(16);
        CHECK(frees == 3 && live.empty());
        frees = 0;
    }
    {   // a buffer that may be in use is freed, not handed on
        CwkBufferPool pool;
        void *a = nullptr;
        size_t na = 0;
        pool.add_context(0);
        pool.alloc(0, MB, &a, &na);
        pool.free(0, a, na, false);
        CHECK(frees == 1 && live.empty());
        frees = 0;
    }
    {   // at most POOL_BYTES wait
        CwkBufferPool pool;
        pool.add_context(0);
        constexpr int fit = CwkBufferPool::POOL_BYTES / (60 * MB), all = fit + 2;
        void *p[all];
        size_t n[all];
        for (int i = 0; i < all; i++) pool.alloc(0, 60 * MB, &p[i], &n[i]);
        for (int i = 0; i < all; i++) pool.free(0, p[i], n[i], true);
        CHECK(live.size() == fit && frees == 2);
        pool.drop_context(0);
        CHECK(live.empty());
        frees = 0;
    }
    {   // what waits is given back before an allocation fails, and a failure leaves the caller's record alone
        CwkBufferPool pool;
        pool.add_context(0);
        memory = 300 * MB;
        void *a = nullptr;
        size_t n = 0;
        pool.alloc(0, 200 * MB, &a, &n);
        pool.free(0, a, n, true);
        a = nullptr;
        n = 0;
        CHECK(pool.alloc(0, 250 * MB, &a, &n) == cudaSuccess && n == 250 * MB && frees == 1);
        void *b = nullptr;
        size_t nb = 0;
        CHECK(pool.alloc(0, 100 * MB, &b, &nb) == cudaErrorMemoryAllocation && b == nullptr && nb == 0);
        pool.free(0, a, n, false);
        pool.drop_context(0);
        memory = SIZE_MAX;
        frees = 0;
    }
    {   // when a context's buffers count as idle
        CwkBufferUse u;
        u.use(stream);
        CHECK(u.known() && u.idle(stream) && syncs == 1);
        sync_fails = true;
        CHECK(!u.idle(stream) && syncs == 2);
        sync_fails = false;
        query_fails = true;                                                  // the legacy stream beside another thread's capture
        u.use(stream);
        CHECK(u.known() && !u.idle(stream) && syncs == 2);
        query_fails = false;
        capture = cudaStreamCaptureStatusActive;                             // not waited for inside a capture
        CHECK(!u.idle(stream) && syncs == 2);
        u.use(stream);                                                       // and once captured, a graph may run it anywhere
        capture = cudaStreamCaptureStatusNone;
        CHECK(!u.known() && !u.idle(stream) && syncs == 2);
        CwkBufferUse v;
        v.lose();
        CHECK(!v.idle(stream) && syncs == 2);
    }
    {   // several threads: no buffer in two hands
        CwkBufferPool pool;
        pool.add_context(0);
        std::mutex mu;
        std::set<void *> held;
        bool twice = false;
        std::vector<std::thread> t;
        for (int k = 0; k < 8; k++)
            t.emplace_back([&] {
                for (int i = 0; i < 2000; i++) {
                    void *p = nullptr;
                    size_t n = 0;
                    pool.alloc(0, MB, &p, &n);
                    { std::lock_guard<std::mutex> l(mu); twice |= !held.insert(p).second; }
                    { std::lock_guard<std::mutex> l(mu); held.erase(p); }
                    pool.free(0, p, n, (i & 7) != 0);
                }
            });
        for (auto &x : t) x.join();
        pool.drop_context(0);
        CHECK(!twice && live.empty());
    }
    puts("ok");
    return 0;
}
