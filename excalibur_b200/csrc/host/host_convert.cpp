#include "host_convert.hpp"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <system_error>

#if defined(__x86_64__) || defined(__i386__)
#include <immintrin.h>
#define EXB_X86 1
#endif

namespace glasssix {
namespace excalibur {

uint16_t f32_to_f16_rne(float v) {
    uint32_t x;
    std::memcpy(&x, &v, 4);
    const uint32_t sign = (x >> 16) & 0x8000u;
    x &= 0x7fffffffu;
    if (x >= 0x7f800000u) return (uint16_t)(sign | (x > 0x7f800000u ? 0x7e00u : 0x7c00u));   // NaN, infinity
    if (x >= 0x47800000u) return (uint16_t)(sign | 0x7c00u);                                   // >= 65536
    if (x < 0x38800000u) {
        // below the smallest normal half (2^-14): adding 0.5f aligns the value's bits with the half's
        // subnormal mantissa in the low bits of the sum, and the float addition rounds to nearest even
        float f;
        std::memcpy(&f, &x, 4);
        f += 0.5f;
        uint32_t y;
        std::memcpy(&y, &f, 4);
        return (uint16_t)(sign | (y - 0x3f000000u));
    }
    // normal: re-bias the exponent (127 -> 15) and round the 13 dropped mantissa bits to nearest even;
    // a carry out of the mantissa moves into the exponent, up to infinity for values >= 65520
    const uint32_t odd = (x >> 13) & 1u;
    x += ((uint32_t)(15 - 127) << 23) + 0xfffu + odd;
    return (uint16_t)(sign | (x >> 13));
}

#ifdef EXB_X86
__attribute__((target("avx,f16c"))) static void convert_f16c(const float* src, uint16_t* dst, size_t n) {
    size_t i = 0;
    for (; i + 16 <= n; i += 16) {
        const __m256 a = _mm256_loadu_ps(src + i), b = _mm256_loadu_ps(src + i + 8);
        _mm_storeu_si128(reinterpret_cast<__m128i*>(dst + i), _mm256_cvtps_ph(a, _MM_FROUND_TO_NEAREST_INT | _MM_FROUND_NO_EXC));
        _mm_storeu_si128(reinterpret_cast<__m128i*>(dst + i + 8),
                         _mm256_cvtps_ph(b, _MM_FROUND_TO_NEAREST_INT | _MM_FROUND_NO_EXC));
    }
    for (; i < n; ++i) dst[i] = f32_to_f16_rne(src[i]);
}
bool host_has_f16c() {
    static const bool has = __builtin_cpu_supports("f16c") && __builtin_cpu_supports("avx");
    return has;
}
#else
bool host_has_f16c() { return false; }
#endif

void convert_f32_to_f16(const float* src, uint16_t* dst, size_t n, bool force_scalar) {
#ifdef EXB_X86
    if (!force_scalar && host_has_f16c()) {
        convert_f16c(src, dst, n);
        return;
    }
#endif
    (void)force_scalar;
    for (size_t i = 0; i < n; ++i) dst[i] = f32_to_f16_rne(src[i]);
}

convert_pool::convert_pool(int threads) {
    if (threads < 1) threads = 1;
    for (int t = 1; t < threads; ++t) workers_.emplace_back([this, t] { worker(t); });
}

convert_pool::~convert_pool() {
    {
        std::lock_guard<std::mutex> lk(mu_);
        stop_ = true;
    }
    start_cv_.notify_all();
    for (auto& w : workers_) w.join();
}

void convert_pool::slice(int index, int parts) {
    // ranges start on multiples of 16 values so every thread but the last runs whole vectors
    const size_t per = (n_ / parts) & ~(size_t)15;
    const size_t a = per * index, b = index == parts - 1 ? n_ : per * (index + 1);
    if (b > a) convert_f32_to_f16(src_ + a, dst_ + a, b - a);
}

void convert_pool::worker(int index) {
    uint64_t seen = 0;
    for (;;) {
        {
            std::unique_lock<std::mutex> lk(mu_);
            start_cv_.wait(lk, [&] { return stop_ || generation_ != seen; });
            if (stop_) return;
            seen = generation_;
        }
        slice(index, threads());
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (--pending_ == 0) done_cv_.notify_one();
        }
    }
}

void convert_pool::run(const float* src, uint16_t* dst, size_t n) {
    const int parts = threads();
    {
        std::lock_guard<std::mutex> lk(mu_);
        src_ = src;
        dst_ = dst;
        n_ = n;
        pending_ = parts - 1;
        ++generation_;
    }
    start_cv_.notify_all();
    slice(0, parts);
    std::unique_lock<std::mutex> lk(mu_);
    done_cv_.wait(lk, [&] { return pending_ == 0; });
}

namespace {
constexpr size_t kCopyBlock = 128 << 10;

// Copy for a device to read: stores that bypass the caches.  A device that reads lines which sit modified in some core's
// cache gets 9 GB/s of 55 (9.6 MB to the GPU in 1.1 ms).
#ifdef EXB_X86
__attribute__((target("avx"))) void copy_streaming_avx(char* dst, const char* src, size_t n) {
    size_t i = 0;
    for (; i < n && (reinterpret_cast<uintptr_t>(dst + i) & 31); ++i) dst[i] = src[i];
    for (; i + 128 <= n; i += 128) {
        const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i));
        const __m256i b = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i + 32));
        const __m256i c = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i + 64));
        const __m256i d = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i + 96));
        _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i), a);
        _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i + 32), b);
        _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i + 64), c);
        _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i + 96), d);
    }
    _mm_sfence();
    if (i < n) std::memcpy(dst + i, src + i, n - i);
}
#endif
void copy_streaming(char* dst, const char* src, size_t n) {
#ifdef EXB_X86
    static const bool avx = __builtin_cpu_supports("avx");
    if (avx) {
        copy_streaming_avx(dst, src, n);
        return;
    }
#endif
    std::memcpy(dst, src, n);
}

class copy_pool {
public:
    explicit copy_pool(int threads) : pid_(getpid()) {
        workers_.reserve(threads);
        try {
            for (int t = 1; t < threads; ++t) workers_.emplace_back([this] { work(); });
        } catch (const std::system_error&) {      // the process may not have more: those there are do the work
        }
    }
    ~copy_pool() {
        if (getpid() != pid_) {      // a forked child has no workers to join
            for (auto& w : workers_) w.detach();
            return;
        }
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto& w : workers_) w.join();
    }
    bool try_copy(char* dst, const char* src, size_t bytes, const std::function<void(size_t)>& ready) {
        if (workers_.empty() || getpid() != pid_ || !turn_.try_lock()) return false;
        std::lock_guard<std::mutex> turn(turn_, std::adopt_lock);
        const size_t blocks = (bytes + kCopyBlock - 1) / kCopyBlock;
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (capacity_ < blocks) {
                complete_.reset(new std::atomic<char>[blocks]);
                capacity_ = blocks;
            }
            for (size_t i = 0; i < blocks; ++i) complete_[i].store(0, std::memory_order_relaxed);
            dst_ = dst;
            src_ = src;
            bytes_ = bytes;
            blocks_ = blocks;
            for_device_ = (bool)ready;
            next_.store(0, std::memory_order_relaxed);
            active_ = 1;
            open_ = true;
        }
        cv_.notify_all();
        // However this call ends - `ready` may throw - no worker is left with the caller's buffers.
        struct closer {
            copy_pool& p;
            ~closer() {
                p.next_.store(p.blocks_, std::memory_order_relaxed);
                std::unique_lock<std::mutex> lk(p.mu_);
                p.open_ = false;                     // a worker that wakes up now finds nothing to do
                --p.active_;
                p.done_.wait(lk, [&] { return p.active_ == 0; });
            }
        } close{*this};
        size_t sent = 0;
        auto report = [&] {
            size_t upto = sent;
            while (upto < blocks && complete_[upto].load(std::memory_order_acquire)) ++upto;
            if (upto > sent && ready) ready(std::min(bytes, upto * kCopyBlock));
            sent = upto;
        };
        while (one()) report();
        while (sent < blocks) {              // the last blocks are in other hands: they are a few microseconds away
            report();
            std::this_thread::yield();
        }
        return true;
    }

private:
    // Copies the next block; blocks are handed out one by one, so that a worker that wakes up late takes less.
    bool one() {
        const size_t i = next_.fetch_add(1, std::memory_order_relaxed);
        if (i >= blocks_) return false;
        const size_t at = i * kCopyBlock, n = std::min(kCopyBlock, bytes_ - at);
        if (for_device_) copy_streaming(dst_ + at, src_ + at, n);
        else std::memcpy(dst_ + at, src_ + at, n);
        complete_[i].store(1, std::memory_order_release);
        return true;
    }
    void work() {
        std::unique_lock<std::mutex> lk(mu_);
        for (;;) {
            cv_.wait(lk, [&] { return stop_ || (open_ && next_.load(std::memory_order_relaxed) < blocks_); });
            if (stop_) return;
            ++active_;
            lk.unlock();
            while (one()) {
            }
            lk.lock();
            if (--active_ == 0) done_.notify_one();
        }
    }
    const pid_t pid_;
    std::vector<std::thread> workers_;
    std::mutex turn_, mu_;
    std::condition_variable cv_, done_;
    std::unique_ptr<std::atomic<char>[]> complete_;
    char* dst_ = nullptr;
    const char* src_ = nullptr;
    size_t bytes_ = 0, blocks_ = 0, capacity_ = 0;
    std::atomic<size_t> next_{0};
    int active_ = 0;
    bool open_ = false, stop_ = false, for_device_ = false;
};
}  // namespace

void host_copy(void* dst, const void* src, size_t bytes, const std::function<void(size_t)>& ready) {
    char* d = static_cast<char*>(dst);
    const char* s = static_cast<const char*>(src);
    if (bytes >= (1 << 20)) {
        static copy_pool pool(std::max(1, std::min(8, (int)std::thread::hardware_concurrency() / 2)));
        if (pool.try_copy(d, s, bytes, ready)) return;
    }
    if (!ready) {
        std::memcpy(d, s, bytes);
        return;
    }
    for (size_t at = 0; at < bytes; at += kCopyBlock) {
        const size_t n = std::min(kCopyBlock, bytes - at);
        copy_streaming(d + at, s + at, n);
        ready(at + n);
    }
}

}  // namespace excalibur
}  // namespace glasssix
