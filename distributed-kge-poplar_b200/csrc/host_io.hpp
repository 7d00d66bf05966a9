// Host side of the transfers: a few helper threads that share the copying between the caller's arrays and pinned
// memory, and the pinned blocks themselves.
#pragma once

#include <cuda_runtime.h>
#include <immintrin.h>
#include <stdint.h>

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include "common.hpp"
#include "pdl.cuh"

namespace kge {

// One core copies 5 GB/s into memory that has not been touched yet (page faults included), a tenth of what the link to
// the GPU moves.  A job is cut into parts that the caller and up to kHelpers threads take in turn; the threads start
// with the first job and end with their owner.  For long transfers only: waking a sleeping helper takes longer than
// copying a megabyte (a 2 MB read takes 400 us with helpers and 150 us without).
class HostTeam {
   public:
    ~HostTeam() {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            stop_ = true;
        }
        wake_.notify_all();
        for (std::thread& t : threads_) t.join();
    }
    // f(part) for every part in [0, parts), in any order; returns when all are done.
    template <class F>
    void run(unsigned parts, F&& f) {
        if (parts <= 1) {
            for (unsigned p = 0; p < parts; ++p) f(p);
            return;
        }
        start();
        struct Call {
            static void one(void* context, unsigned part) { (*static_cast<std::remove_reference_t<F>*>(context))(part); }
        };
        {
            std::lock_guard<std::mutex> lock(mutex_);
            work_ = &Call::one;
            context_ = &f;
            parts_ = parts;
            next_.store(0, std::memory_order_relaxed);
            active_ = 0;
            ++generation_;
            seen_.store(generation_, std::memory_order_release);
        }
        wake_.notify_all();
        take_parts(&Call::one, &f, parts);
        // no part is left to take; wait for the helpers that still work on one
        std::unique_lock<std::mutex> lock(mutex_);
        work_ = nullptr;
        done_.wait(lock, [this] { return active_ == 0; });
    }

   private:
    static constexpr unsigned kHelpers = 7;
    using Work = void (*)(void*, unsigned);

    void take_parts(Work work, void* context, unsigned parts) {
        for (unsigned p; (p = next_.fetch_add(1, std::memory_order_relaxed)) < parts;) work(context, p);
    }
    void start() {
        if (!threads_.empty()) return;
        const unsigned half = std::thread::hardware_concurrency() / 2, n = half > kHelpers ? kHelpers : (half > 1 ? half - 1 : 0);
        for (unsigned i = 0; i < n; ++i) threads_.emplace_back([this] { helper(); });
    }
    void helper() {
        unsigned long long mine = 0;
        for (;;) {
            // a run of jobs follows each other closely: look for the next one for some 50 us before sleeping
            for (int spin = 0; spin < 2000 && seen_.load(std::memory_order_acquire) == mine; ++spin) __builtin_ia32_pause();
            std::unique_lock<std::mutex> lock(mutex_);
            wake_.wait(lock, [&] { return stop_ || generation_ != mine; });
            if (stop_) return;
            mine = generation_;
            if (!work_) continue;  // that job is over already
            const Work work = work_;
            void* const context = context_;
            const unsigned parts = parts_;
            ++active_;
            lock.unlock();
            take_parts(work, context, parts);
            lock.lock();
            if (--active_ == 0) done_.notify_one();
        }
    }

    std::mutex mutex_;
    std::condition_variable wake_, done_;
    std::vector<std::thread> threads_;
    std::atomic<unsigned> next_{0};
    std::atomic<unsigned long long> seen_{0};
    unsigned long long generation_ = 0;
    Work work_ = nullptr;
    void* context_ = nullptr;
    unsigned parts_ = 0, active_ = 0;
    bool stop_ = false;
};

// Writes a byte of every page of an array that is about to be overwritten whole: fresh memory is mapped and cleared by
// the kernel at the first touch, up to 2 MB at a time, and threads that copy into the same large page wait for one of
// them to clear it.  Here every thread has large pages of its own (123 MB: 13 ms by one thread, 2 ms by eight).
inline void team_touch(HostTeam& team, void* dst, size_t bytes) {
    constexpr size_t kLarge = 2 << 20, kSmall = 4096;
    uint8_t* const begin = static_cast<uint8_t*>(dst);
    const size_t lead = (kLarge - reinterpret_cast<uintptr_t>(begin) % kLarge) % kLarge;  // parts start where large pages do
    team.run((unsigned)(1 + (bytes > lead ? (bytes - lead + kLarge - 1) / kLarge : 0)), [=](unsigned p) {
        const size_t from = p == 0 ? 0 : lead + (size_t)(p - 1) * kLarge, to = p == 0 ? (lead < bytes ? lead : bytes) : (from + kLarge < bytes ? from + kLarge : bytes);
        for (size_t at = from; at < to; at += kSmall) reinterpret_cast<volatile uint8_t*>(begin)[at] = 0;
    });
}

// memcpy whose stores bypass the caches: what a bulk transfer writes is not read again soon, and an ordinary store
// would first fetch the line it overwrites (123 MB out 12 to 9 ms, 61 MB in 4.5 to 3.4 ms).
__attribute__((target("avx2"))) inline void streaming_copy_avx2(uint8_t* d, const uint8_t* s, size_t n) {
    for (; n && (reinterpret_cast<uintptr_t>(d) & 31); --n) *d++ = *s++;
    for (; n >= 128; n -= 128, d += 128, s += 128) {
        const __m256i* in = reinterpret_cast<const __m256i*>(s);
        __m256i* out = reinterpret_cast<__m256i*>(d);
        const __m256i v0 = _mm256_loadu_si256(in), v1 = _mm256_loadu_si256(in + 1), v2 = _mm256_loadu_si256(in + 2), v3 = _mm256_loadu_si256(in + 3);
        _mm256_stream_si256(out, v0);
        _mm256_stream_si256(out + 1, v1);
        _mm256_stream_si256(out + 2, v2);
        _mm256_stream_si256(out + 3, v3);
    }
    _mm_sfence();
    std::memcpy(d, s, n);
}
inline void streaming_copy(uint8_t* d, const uint8_t* s, size_t n) {
    static const bool avx2 = __builtin_cpu_supports("avx2");
    if (avx2) streaming_copy_avx2(d, s, n);
    else std::memcpy(d, s, n);
}

// Copies in parts of 128 KB, with the team's help when there is one.
inline void team_copy(HostTeam* team, void* dst, const void* src, size_t bytes) {
    if (!team) {
        std::memcpy(dst, src, bytes);
        return;
    }
    constexpr size_t kPart = 128 * 1024;
    team->run((unsigned)((bytes + kPart - 1) / kPart), [=](unsigned p) {
        const size_t at = (size_t)p * kPart;
        streaming_copy(static_cast<uint8_t*>(dst) + at, static_cast<const uint8_t*>(src) + at, bytes - at < kPart ? bytes - at : kPart);
    });
}

// Pinned blocks for transfers of the callers' arrays, lent out for the length of a command: pinning memory costs the
// host about a millisecond for a block.  At most kKept blocks (16 MB) wait for the next borrower; the rest are freed.
class PinnedPool {
   public:
    static constexpr size_t kBlock = 4 << 20;
    static PinnedPool& instance() {
        static PinnedPool* pool = new PinnedPool;  // never destroyed: CUDA may be gone before static destructors run
        return *pool;
    }
    uint8_t* take() {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (!free_.empty()) {
                uint8_t* p = free_.back();
                free_.pop_back();
                return p;
            }
        }
        void* p = nullptr;
        KGE_CUDA(cudaHostAlloc(&p, kBlock, cudaHostAllocPortable));
        return static_cast<uint8_t*>(p);
    }
    void give(uint8_t* p) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (free_.size() < kKept) {
                free_.push_back(p);
                return;
            }
        }
        cudaFreeHost(p);
    }

   private:
    static constexpr size_t kKept = 4;
    std::mutex mutex_;
    std::vector<uint8_t*> free_;
};

// Whether a scope is being left by an exception that came up inside it: its transfers may still be under way, so its
// blocks are not lent to anyone else but freed, for which CUDA waits.
class LeftByException {
   public:
    explicit operator bool() const { return std::uncaught_exceptions() > at_entry_; }

   private:
    const int at_entry_ = std::uncaught_exceptions();
};

// A block of the pool for the length of a scope.  Its transfers must have completed when the scope ends as it should.
class PinnedBlock {
   public:
    explicit PinnedBlock(size_t bytes = PinnedPool::kBlock) : pooled_(bytes <= PinnedPool::kBlock) {
        if (pooled_) data_ = PinnedPool::instance().take();
        else KGE_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&data_), bytes, cudaHostAllocPortable));
    }
    ~PinnedBlock() {
        if (pooled_ && !left_by_exception_) PinnedPool::instance().give(data_);
        else cudaFreeHost(data_);
    }
    PinnedBlock(const PinnedBlock&) = delete;
    PinnedBlock& operator=(const PinnedBlock&) = delete;
    uint8_t* data() const { return data_; }

   private:
    LeftByException left_by_exception_;
    bool pooled_;
    uint8_t* data_ = nullptr;
};

// The same on the GPU: a block for the pieces of a transfer in device memory (an allocation costs 0.3 ms), lent out for
// the length of a command; at most kKept per device wait for the next borrower.
class DeviceBlock {
   public:
    static constexpr size_t kBytes = PinnedPool::kBlock;
    DeviceBlock() = default;
    ~DeviceBlock() {
        if (!data_) return;
        if (!left_by_exception_) {
            std::lock_guard<std::mutex> lock(pool().mutex);
            if (slot_ >= 0 && pool().free[slot_].size() < kKept) {
                pool().free[slot_].push_back(data_);
                return;
            }
        }
        cudaFree(data_);
    }
    DeviceBlock(const DeviceBlock&) = delete;
    DeviceBlock& operator=(const DeviceBlock&) = delete;
    uint8_t* get() {  // taken at the first call
        if (data_) return data_;
        slot_ = current_device_slot();
        {
            std::lock_guard<std::mutex> lock(pool().mutex);
            if (slot_ >= 0 && !pool().free[slot_].empty()) {
                data_ = pool().free[slot_].back();
                pool().free[slot_].pop_back();
                return data_;
            }
        }
        KGE_CUDA(cudaMalloc(reinterpret_cast<void**>(&data_), kBytes));
        return data_;
    }

   private:
    static constexpr size_t kKept = 2;
    struct Pool {
        std::mutex mutex;
        std::vector<uint8_t*> free[kMaxDeviceOrdinals];
    };
    static Pool& pool() {
        static Pool* p = new Pool;
        return *p;
    }
    LeftByException left_by_exception_;
    uint8_t* data_ = nullptr;
    int slot_ = -1;
};

// out[i] = in[i]; returns the largest element (0 of none).
__attribute__((target_clones("avx2", "default"))) inline uint32_t copy_and_max(uint32_t* __restrict__ out, const uint32_t* __restrict__ in, size_t n) {
    uint32_t highest = 0;
    for (size_t i = 0; i < n; ++i) {
        const uint32_t v = in[i];
        out[i] = v;
        highest = v > highest ? v : highest;
    }
    return highest;
}

}  // namespace kge
