// hostpix.cpp -- see hostpix.h.
//
// Bound: the read of the pixels from host memory.  A copy of pageable memory to
// the device ran at 20 GB/s (12.2 MB of int16: 0.56-0.65 ms, and another 55 us
// in which the kernel turned them into words); packing them here first leaves
// 1/16 of the bytes for the link.  One thread packs about 12 GB/s of bytes and
// 6 GB/s of floats and unpacks 4 GB/s, hence the rule of host_pack_pays.
#include "hostpix.h"

#include <sched.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include "bgt_capi.h"

namespace bgt {
namespace {

// ------------------------------------------------------------ workers -----
// One job at a time, its parts handed out by a counter; the caller works too.
// A second caller finds the pool busy and does its job alone.
class Pool {
public:
    using Fn = void (*)(void *, int);

    explicit Pool(int threads)
    {
        try {
            for (int i = 0; i < threads; i++) th_.emplace_back([this] { work(); });
        } catch (...) {  // fewer workers than wanted
        }
    }
    ~Pool()
    {
        {
            std::lock_guard<std::mutex> l(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto &t : th_) t.join();
    }
    int size() const { return (int)th_.size(); }
    void run(Fn fn, void *arg, int parts)
    {
        std::unique_lock<std::mutex> busy(busy_, std::try_to_lock);
        if (!busy.owns_lock() || th_.empty()) {
            for (int k = 0; k < parts; k++) fn(arg, k);
            return;
        }
        {
            std::lock_guard<std::mutex> l(m_);
            fn_ = fn;
            arg_ = arg;
            parts_ = parts;
            next_ = 0;
            in_job_ = 0;
            job_++;
        }
        cv_.notify_all();
        for (int k; (k = next_.fetch_add(1)) < parts;) fn(arg, k);
        // no worker joins any more once parts are out; wait for those inside
        std::unique_lock<std::mutex> l(m_);
        fn_ = nullptr;
        done_.wait(l, [this] { return in_job_ == 0; });
    }

private:
    void work()
    {
        unsigned long long seen = 0;
        std::unique_lock<std::mutex> l(m_);
        for (;;) {
            cv_.wait(l, [&] { return stop_ || (fn_ && job_ != seen); });
            if (stop_) return;
            seen = job_;
            const Fn fn = fn_;
            void *const arg = arg_;
            const int parts = parts_;
            in_job_++;
            l.unlock();
            for (int k; (k = next_.fetch_add(1)) < parts;) fn(arg, k);
            l.lock();
            if (--in_job_ == 0) done_.notify_all();
        }
    }
    std::vector<std::thread> th_;
    std::mutex m_, busy_;
    std::condition_variable cv_, done_;
    Fn fn_ = nullptr;
    void *arg_ = nullptr;
    int parts_ = 0, in_job_ = 0;
    std::atomic<int> next_{0};
    unsigned long long job_ = 0;
    bool stop_ = false;
};

std::mutex g_pool_m;
Pool *g_pool = nullptr;  // never destroyed at exit: contexts may outlive static objects
pid_t g_pool_pid = 0;
int g_users = 0;

// The pool, started on first use (null: none).  A process forked from one that
// had a pool starts its own.
Pool *pool()
{
    std::lock_guard<std::mutex> l(g_pool_m);
    if (g_users > 0 && (!g_pool || g_pool_pid != getpid())) {
        cpu_set_t set;
        CPU_ZERO(&set);
        const int cpus = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : 1;
        try {
            g_pool = cpus > 1 ? new Pool(std::min(cpus, 8) - 1) : nullptr;
        } catch (...) {
            g_pool = nullptr;
        }
        g_pool_pid = getpid();
    }
    return g_pool;
}

constexpr size_t kPartBytes = 256 << 10;  // a part of a job; one part is done by the caller alone

// fn(arg, part) over `parts` parts
void run_parts(Pool::Fn fn, void *arg, int parts)
{
    Pool *p = parts > 1 ? pool() : nullptr;
    if (p) {
        p->run(fn, arg, parts);
        return;
    }
    for (int k = 0; k < parts; k++) fn(arg, k);
}

// ------------------------------------------------------------ pack --------
// Foreground tests as the device evaluates them (pixels.cuh).
template <class T, int MODE>
inline bool fg(T v)
{
    if constexpr (std::is_same<T, float>::value || std::is_same<T, double>::value)
        return v >= (T)1 && (MODE == 0 || v < (T)2147483648.0);
    else if constexpr (std::is_same<T, bool>::value)
        return v;
    else
        return MODE == 0 ? v != (T)0 : (int)v > 0;
}

#if defined(__SSE2__)
inline __m128i load16(const void *p) { return _mm_loadu_si128(static_cast<const __m128i *>(p)); }

// 16 pixels -> 16 bits
template <class T, int MODE>
inline uint32_t bits16(const T *p)
{
    const __m128i zero = _mm_setzero_si128();
    if constexpr (sizeof(T) == 1) {
        const __m128i v = load16(p);
        if (MODE == 1 && std::is_signed<T>::value) return (uint32_t)_mm_movemask_epi8(_mm_cmpgt_epi8(v, zero));
        return (uint32_t)_mm_movemask_epi8(_mm_cmpeq_epi8(v, zero)) ^ 0xFFFFu;
    } else if constexpr (sizeof(T) == 2) {
        const __m128i a = load16(p), b = load16(p + 8);
        if (MODE == 1 && std::is_signed<T>::value)
            return (uint32_t)_mm_movemask_epi8(_mm_packs_epi16(_mm_cmpgt_epi16(a, zero), _mm_cmpgt_epi16(b, zero)));
        return (uint32_t)_mm_movemask_epi8(_mm_packs_epi16(_mm_cmpeq_epi16(a, zero), _mm_cmpeq_epi16(b, zero))) ^ 0xFFFFu;
    } else if constexpr (std::is_same<T, float>::value) {
        uint32_t r = 0;
        const __m128 one = _mm_set1_ps(1.0f), top = _mm_set1_ps(2147483648.0f);
        for (int k = 0; k < 4; k++) {
            const __m128 v = _mm_loadu_ps(p + 4 * k);
            __m128 m = _mm_cmpge_ps(v, one);
            if (MODE == 1) m = _mm_and_ps(m, _mm_cmplt_ps(v, top));
            r |= (uint32_t)_mm_movemask_ps(m) << (4 * k);
        }
        return r;
    } else if constexpr (std::is_same<T, double>::value) {
        uint32_t r = 0;
        const __m128d one = _mm_set1_pd(1.0), top = _mm_set1_pd(2147483648.0);
        for (int k = 0; k < 8; k++) {
            const __m128d v = _mm_loadu_pd(p + 2 * k);
            __m128d m = _mm_cmpge_pd(v, one);
            if (MODE == 1) m = _mm_and_pd(m, _mm_cmplt_pd(v, top));
            r |= (uint32_t)_mm_movemask_pd(m) << (2 * k);
        }
        return r;
    } else {
        uint32_t r = 0;
        for (int k = 0; k < 4; k++) {
            const __m128i v = load16(p + 4 * k);
            // 3D: (int)v > 0, also for unsigned pixels
            const __m128i m = MODE == 1 ? _mm_cmpgt_epi32(v, zero) : _mm_cmpeq_epi32(v, zero);
            r |= (uint32_t)_mm_movemask_ps(_mm_castsi128_ps(m)) << (4 * k);
        }
        return MODE == 1 ? r : r ^ 0xFFFFu;
    }
}
#endif

template <class T, int MODE>
void pack_row(const T *p, int w, int P, uint32_t *out)
{
    int j = 0;
#if defined(__SSE2__)
    for (; 32 * j + 32 <= w; j++) out[j] = bits16<T, MODE>(p + 32 * j) | bits16<T, MODE>(p + 32 * j + 16) << 16;
#endif
    for (; 32 * j < w; j++) {
        uint32_t v = 0;
        for (int b = 0; b < 32 && 32 * j + b < w; b++) v |= (uint32_t)fg<T, MODE>(p[32 * j + b]) << b;
        out[j] = v;
    }
    for (; j < P; j++) out[j] = 0;
}

struct PackJob {
    const void *in;
    int w, h, d, H, D, P, parts;
    uint32_t *out;
    void (*rows)(const PackJob &, long long, long long);
};

template <class T, int MODE>
void pack_rows(const PackJob &j, long long r0, long long r1)
{
    for (long long r = r0; r < r1; r++) {
        const int y = (int)(r % j.H);
        const long long z = r / j.H;
        uint32_t *o = j.out + r * j.P;
        if (y < j.h && z < j.d) pack_row<T, MODE>(static_cast<const T *>(j.in) + (z * j.h + y) * j.w, j.w, j.P, o);
        else memset(o, 0, (size_t)j.P * 4);
    }
}

void pack_part(void *arg, int k)
{
    const PackJob &j = *static_cast<const PackJob *>(arg);
    const long long rows = (long long)j.H * j.D;
    j.rows(j, rows * k / j.parts, rows * (k + 1) / j.parts);
}

// ------------------------------------------------------------ unpack ------
// N values of each of the 2^N bit patterns
template <class T, int N>
struct Table {
    T v[1 << N][N];
    Table()
    {
        for (int i = 0; i < 1 << N; i++)
            for (int b = 0; b < N; b++) v[i][b] = (T)((i >> b) & 1);
    }
};

struct UnpackJob {
    const uint32_t *words;
    int w, h, d, P, parts;
    void *out;
    void (*rows)(const UnpackJob &, long long, long long);
};

template <class T>
void unpack_rows(const UnpackJob &j, long long r0, long long r1)
{
    constexpr int N = sizeof(T) == 1 ? 8 : 4;
    static const Table<T, N> t;
    for (long long r = r0; r < r1; r++) {
        const uint32_t *s = j.words + r * j.P;
        T *o = static_cast<T *>(j.out) + r * j.w;
        int x = 0;
        for (; x + 32 <= j.w; x += 32) {
            const uint32_t v = s[x >> 5];
            for (int k = 0; k < 32; k += N) memcpy(o + x + k, t.v[(v >> k) & ((1u << N) - 1u)], N * sizeof(T));
        }
        for (; x < j.w; x++) o[x] = (T)((s[x >> 5] >> (x & 31)) & 1u);
    }
}

void unpack_part(void *arg, int k)
{
    const UnpackJob &j = *static_cast<const UnpackJob *>(arg);
    const long long rows = (long long)j.h * j.d;
    j.rows(j, rows * k / j.parts, rows * (k + 1) / j.parts);
}

int parts_of(size_t bytes, long long rows)
{
    return (int)std::max<long long>(1, std::min<long long>({(long long)(bytes / kPartBytes), rows, 64}));
}

template <template <class> class F, class R>
R by_type(int dtype)
{
    switch (dtype) {
    case BGT_U8: return F<uint8_t>::get();
    case BGT_I8: return F<int8_t>::get();
    case BGT_CHAR: return F<char>::get();
    case BGT_U16: return F<uint16_t>::get();
    case BGT_I16: return F<int16_t>::get();
    case BGT_U32: return F<uint32_t>::get();
    case BGT_I32: return F<int32_t>::get();
    case BGT_F32: return F<float>::get();
    case BGT_F64: return F<double>::get();
    default: return F<bool>::get();
    }
}
using PackRows = void (*)(const PackJob &, long long, long long);
using UnpackRows = void (*)(const UnpackJob &, long long, long long);
// bool pixels are bytes that are zero or not
template <class T>
using Stored = typename std::conditional<std::is_same<T, bool>::value, uint8_t, T>::type;
template <class T>
struct Pack2 {
    static PackRows get() { return pack_rows<Stored<T>, 0>; }
};
template <class T>
struct Pack3 {
    static PackRows get() { return pack_rows<Stored<T>, 1>; }
};
template <class T>
struct Unpack {
    static UnpackRows get() { return unpack_rows<Stored<T>>; }
};
template <class T>
struct Size {
    static size_t get() { return sizeof(T); }
};
}  // namespace

void host_pack(int dtype, int mode, const void *in, int w, int h, int d, int H, int D, int P, uint32_t *out)
{
    PackJob j{in, w, h, d, H, D, P, 1, out, mode == 0 ? by_type<Pack2, PackRows>(dtype) : by_type<Pack3, PackRows>(dtype)};
    j.parts = parts_of((size_t)w * h * d * by_type<Size, size_t>(dtype), (long long)H * D);
    run_parts(pack_part, &j, j.parts);
}

void host_unpack(int dtype, const uint32_t *words, int w, int h, int d, int P, void *out)
{
    UnpackJob j{words, w, h, d, P, 1, out, by_type<Unpack, UnpackRows>(dtype)};
    j.parts = parts_of((size_t)w * h * d * by_type<Size, size_t>(dtype), (long long)h * d);
    run_parts(unpack_part, &j, j.parts);
}

bool host_pack_pays(size_t pixel, size_t bytes, bool pinned, int workers)
{
    return pinned ? pixel >= 4 && workers >= 3 : pixel >= 4 || bytes <= (2u << 20) || workers >= 1;
}

int host_workers()
{
    Pool *p = pool();
    return p ? p->size() : 0;
}

void host_pool_retain()
{
    std::lock_guard<std::mutex> l(g_pool_m);
    g_users++;
}

void host_pool_release()
{
    Pool *gone = nullptr;
    {
        std::lock_guard<std::mutex> l(g_pool_m);
        if (--g_users == 0 && g_pool && g_pool_pid == getpid()) {
            gone = g_pool;
            g_pool = nullptr;
        }
    }
    delete gone;
}

}  // namespace bgt
