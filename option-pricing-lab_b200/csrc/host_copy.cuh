// Copies of device results into the caller's pageable host arrays. A device-to-host copy into pageable memory runs at
// the driver's single-threaded staging rate (117 MB of path columns: 6.7 ms on a B200 host); into pinned memory it
// runs at the link's rate (2.2 ms), and host threads then spread the bytes into the caller's array in parallel.
// Pinning the caller's array itself costs more than the copy (117 MB: 12.5 ms), so the library keeps its own pinned
// staging, two slots reused from call to call.
#pragma once

#include <algorithm>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>

#include "common.cuh"

#if defined(__x86_64__)
#include <cpuid.h>
#include <emmintrin.h>
#include <immintrin.h>
#endif

namespace ob {

// Host memory that the GPU's copy engine reads or overwrites should not sit in the caches of the cores that wrote or
// read it: on a B200 host a 4.8 MB upload takes 100 us from memory, and 750 us from lines dirty in eight cores' caches;
// 11 MB of results land in 207 us, in 480 to 1300 us over lines those cores hold. So the threads write the staging
// past the caches (stream_copy), and give up the lines they have read from it (drop_lines).
// Copies n bytes to a 16-byte-aligned dst with non-temporal stores (src as aligned as dst).
inline void stream_copy(void* dst, const void* src, size_t n) {
#if defined(__x86_64__)
    const size_t whole = n / 16;
    const __m128i* s = static_cast<const __m128i*>(src);
    __m128i* d = static_cast<__m128i*>(dst);
    for (size_t i = 0; i < whole; ++i) _mm_stream_si128(d + i, _mm_loadu_si128(s + i));
    std::memcpy(d + whole, s + whole, n - 16 * whole);
    _mm_sfence();
#else
    std::memcpy(dst, src, n);
#endif
}
#if defined(__x86_64__)
__attribute__((target("clflushopt"))) inline void drop_lines_opt(const char* p, size_t n) {
    for (size_t i = 0; i < n; i += 64) _mm_clflushopt(const_cast<char*>(p + i));
    _mm_sfence();
}
#endif
inline void drop_lines(const void* p, size_t n) {
#if defined(__x86_64__)
    static const bool have = [] {
        unsigned a = 0, b = 0, c = 0, d = 0;
        return __get_cpuid_count(7, 0, &a, &b, &c, &d) && ((b >> 23) & 1u);  // CLFLUSHOPT
    }();
    if (have) drop_lines_opt(static_cast<const char*>(p), n);
#else
    (void)p, (void)n;
#endif
}
// n values of T widened into out (doubles), written past the caches where out allows it (8-byte aligned memory of which
// every second double is 16-byte aligned).
template <typename T>
inline void widen(double* out, const T* from, long long n) {
    long long k = 0;
#if defined(__x86_64__)
    if (n > 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 8u) out[0] = static_cast<double>(from[0]), k = 1;
    if ((reinterpret_cast<uintptr_t>(out) & 7u) == 0u) {
        for (; k + 2 <= n; k += 2)
            _mm_stream_pd(out + k, _mm_set_pd(static_cast<double>(from[k + 1]), static_cast<double>(from[k])));
        _mm_sfence();
    }
#endif
    for (; k < n; ++k) out[k] = static_cast<double>(from[k]);
}

// Two pinned slots, allocated at their first use and kept until release() (ob_release_buffers): of kSmallBytes while
// that is enough, else of kSlotBytes (pinning costs 0.4 ms a megabyte, so a process that only uploads a table does not pay
// for the path engine's). Portable pinned memory: any device's copies may use it. The library's calls are serialised and
// finish their copies before they return, so a larger pair may replace the smaller one at the next call.
class PinnedStage {
  public:
    static constexpr size_t kSmallBytes = size_t(4) << 20, kSlotBytes = size_t(32) << 20;
    static PinnedStage& get() {
        static PinnedStage* s = new PinnedStage();
        return *s;
    }
    // Both slots with room for `need` bytes each (at most kSlotBytes); false where pinned memory cannot be had (the
    // caller then copies from or into pageable memory).
    bool slots(size_t need, char* (&out)[2]) {
        std::lock_guard<std::mutex> lock(m_);
        const size_t want = need <= kSmallBytes ? kSmallBytes : kSlotBytes;
        if (need > kSlotBytes) return false;
        if (size_ < want && want < refused_) {
            void* more = nullptr;
            if (cudaHostAlloc(&more, 2 * want, cudaHostAllocPortable) == cudaSuccess) {
                if (base_) cudaFreeHost(base_);
                base_ = more, size_ = want;
            } else {
                cudaGetLastError();
                refused_ = want;  // a smaller pair, held or not, still serves
            }
        }
        if (size_ < want) return false;
        out[0] = static_cast<char*>(base_), out[1] = static_cast<char*>(base_) + size_;
        return true;
    }
    void release() {
        std::lock_guard<std::mutex> lock(m_);
        if (base_) cudaFreeHost(base_);
        cudaGetLastError();
        base_ = nullptr, size_ = 0, refused_ = ~size_t(0);
    }

  private:
    std::mutex m_;
    void* base_ = nullptr;
    size_t size_ = 0;
    size_t refused_ = ~size_t(0);  // the smallest slots that could not be had
};

// Host threads for the copies out of the staging: the hardware threads less one, at most seven, started at the first
// use and kept for the process (never joined: they wait on a condition variable between jobs).
class HostPool {
  public:
    static HostPool& get() {
        static HostPool* p = new HostPool();
        return *p;
    }
    // fn(i) for every i in [0, n), on the pool's threads and the calling one; returns when every call has returned.
    void run(int n, const std::function<void(int)>& fn) {
        if (n <= 0) return;
        std::lock_guard<std::mutex> one(run_m_);
        unsigned long long g;
        {
            std::lock_guard<std::mutex> lock(m_);
            fn_ = &fn, n_ = n, next_ = 0, done_ = 0;
            g = ++gen_;
        }
        cv_.notify_all();
        work(g);
        std::unique_lock<std::mutex> lock(m_);
        done_cv_.wait(lock, [&] { return done_ == n_; });
        fn_ = nullptr;
    }

  private:
    HostPool() {
        const int hw = static_cast<int>(std::thread::hardware_concurrency());
        const int n = std::max(0, std::min(7, hw - 1));
        for (int k = 0; k < n; ++k) std::thread([this] { loop(); }).detach();
    }
    void loop() {
        unsigned long long seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lock(m_);
                cv_.wait(lock, [&] { return gen_ != seen; });
                seen = gen_;
            }
            work(seen);
        }
    }
    // Items of job g, one at a time under the lock, until none is left (or another job has begun).
    void work(unsigned long long g) {
        for (;;) {
            int i;
            const std::function<void(int)>* fn;
            {
                std::lock_guard<std::mutex> lock(m_);
                if (gen_ != g || next_ >= n_) return;
                i = next_++, fn = fn_;
            }
            (*fn)(i);
            std::lock_guard<std::mutex> lock(m_);
            if (++done_ == n_) done_cv_.notify_all();
        }
    }
    std::mutex run_m_, m_;
    std::condition_variable cv_, done_cv_;
    const std::function<void(int)>* fn_ = nullptr;
    int n_ = 0, next_ = 0, done_ = 0;
    unsigned long long gen_ = 0;
};

// n bytes to dst on the device through the two pinned slots: make(out, at, count) writes bytes [at, at + count) of the
// source into out, for blocks of 4 KB at multiples of 4 KB (so a source of records of 8 or 16 bytes converts block by
// block) spread over the host threads; a slot's copy runs while the other is filled. The copies have finished when it
// returns. False (nothing done) below kStagedUpload bytes, where one pageable copy is as fast, and without pinned memory.
template <typename Make>
bool staged_upload(char* dst, size_t n, Make make) {
    if (n < kStagedUpload) return false;
    const size_t slot_bytes = n <= 4 * PinnedStage::kSmallBytes ? PinnedStage::kSmallBytes : PinnedStage::kSlotBytes;
    char* slot[2];
    if (!PinnedStage::get().slots(slot_bytes, slot)) return false;
    constexpr size_t kPiece = size_t(256) << 10, kBlock = 4096;
    cudaStream_t st = kept_stream(2);
    int k = 0;
    for (size_t at = 0; at < n; at += slot_bytes, ++k) {
        if (k > 1) check_cuda(cudaStreamSynchronize(st), "cudaStreamSynchronize (inputs)");  // slot k % 2 is free
        const size_t count = std::min(slot_bytes, n - at);
        char* out = slot[k % 2];
        HostPool::get().run(static_cast<int>((count + kPiece - 1) / kPiece), [&](int item) {
            alignas(64) char block[kBlock];
            const size_t p0 = static_cast<size_t>(item) * kPiece, p1 = std::min(count, p0 + kPiece);
            for (size_t q = p0; q < p1; q += kBlock) {
                const size_t m = std::min(kBlock, p1 - q);
                make(block, at + q, m);
                stream_copy(out + q, block, m);
            }
        });
        check_cuda(cudaMemcpyAsync(dst + at, out, count, cudaMemcpyHostToDevice, st), "cudaMemcpyAsync (inputs)");
    }
    check_cuda(cudaStreamSynchronize(st), "cudaStreamSynchronize (inputs)");
    return true;
}

}  // namespace ob
