// Copies between the device and pageable host memory, by way of page-locked pieces that several threads fill or empty.
//
// The driver copies pageable memory through a buffer of its own with one thread: 3 MB in 200 us, 24 MB in 1.2 to 1.4 ms, either
// way, where the link needs 55 us and 430 (page-locked memory). One core's memcpy is the limit (18 GB/s). Here the caller and up
// to three helpers copy parts of pieces of 512 KB, and a piece is on the link while the next ones are being filled.
//
// A transfer holds a set of pieces from the first copy that is queued on, and the helpers only while there is something to copy: what
// the stream still computes in front of a result keeps nobody busy. One transfer at a time has the helpers; others, meanwhile, copy
// their pieces alone. Small copies (all that is ever recorded into a graph here is small), page-locked memory, callers that have no
// second core for a helper, and whoever finds all sets held take the driver's way. Nothing waits for a helper that has not taken a part
// yet: without helpers (none could be started, a forked child) the caller copies all of it. Threads that wait for one another look
// for a bounded time, then they sleep: the one that is waited for may need their core.
#include "hostcopy.h"

#include <sched.h>
#include <stdio.h>
#include <string.h>
#include <unistd.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <memory>
#include <mutex>
#include <thread>

namespace mb {
namespace {

constexpr size_t PIECE = 512 << 10, PART = 64 << 10;
constexpr int SLOTS = 4;                                         // page-locked pieces of a set: 2 MB (page-locking takes 1 ms per MB, once)
constexpr int SETS = 4;                                          // made when as many transfers are under way at once
// Us of a call with 3 MB of rows and 0.8 MB of results (and of processor time): two helpers 192 (440), three 183 (510), the driver's way
// 305 (310); with 24 and 6 MB 1226 (3480), 1030 (3780), 2650 (2680).
constexpr int HELPERS = 3;
// Waking a thread takes 17 us there, and a part 3.5: a helper that sleeps is not woken for the last FRESH parts.
constexpr int FRESH = 3;
// How long a thread looks within a transfer before it sleeps (with 25 us instead, four processes that shared a device took 8 ms instead of
// 2.5 for a call of 24 and 6 MB: their pieces wait for one another on the link), and how long a helper looks out for the next
// transfer (the smaller call, with 2 ms in front: 5 us 210, 10 us 199, 20 us 199, at 537, 531 and 592 us of processor time).
constexpr auto PATIENCE = std::chrono::microseconds(200), LOOK = std::chrono::microseconds(10);
// Below these the driver's way is as fast, or faster when the helpers are asleep. Us of a product whose rows (results) are so large,
// new memory each time, driver and pieces, with no pause between calls and with 2 ms:
//   in   0.5 MB  91, 85; 96, 101    0.63 MB  102, 97; 106, 108    0.75 MB  110, 100; 115, 112    1 MB  139, 110; 144, 121
//   out  0.5 MB  81, 56; 84,  81    0.63 MB   90, 62;  90,  94    0.75 MB   96,  68;  96,  97    1 MB  113,  86; 120, 115
constexpr size_t LEAST_IN = 640 << 10, LEAST_OUT = 512 << 10;
constexpr int PARTS = (int)(PIECE / PART);

// what a thread does between two looks at a word that another one writes
inline void cpu_relax() {
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#elif defined(__aarch64__)
    asm volatile("yield" ::: "memory");
#else
    std::this_thread::yield();
#endif
}
template <typename F> bool spin(std::chrono::microseconds limit, F ready) {
    const auto until = std::chrono::steady_clock::now() + limit;
    do
        for (int i = 0; i < 16; i++) {
            if (ready()) return true;
            cpu_relax();
        }
    while (std::chrono::steady_clock::now() < until);
    return false;
}

// Cores' worth of time that the control group of the process may use.
int quota_cores() {
    constexpr int ALL = 1 << 20;
    long long quota = 0, period = 0;
    auto read = [](const char *path, const char *format, long long *a, long long *b) {
        FILE *f = fopen(path, "re");
        if (!f) return 0;
        const int got = fscanf(f, format, a, b);
        fclose(f);
        return got;
    };
    // the group of a container, as it sees itself ("max 100000" where there is no limit); else version 1 ("-1")
    if (read("/sys/fs/cgroup/cpu.max", "%lld %lld", &quota, &period) != 2 &&
        (read("/sys/fs/cgroup/cpu/cpu.cfs_quota_us", "%lld", &quota, nullptr) != 1 || read("/sys/fs/cgroup/cpu/cpu.cfs_period_us", "%lld", &period, nullptr) != 1))
        return ALL;
    return quota > 0 && period > 0 && quota / period < ALL ? (int)(quota / period) : ALL;
}

// Cores that the calling thread and helpers started by it may run on (not those of the machine: with helpers on the caller's own core,
// 3 MB of rows on the link took 14 ms instead of 0.3). Real-time and idle threads count as one: helpers would inherit the class.
int caller_cores(int quota) {
    const int policy = sched_getscheduler(0) & ~SCHED_RESET_ON_FORK;
    if (policy != SCHED_OTHER && policy != SCHED_BATCH) return 1;
    cpu_set_t set[8];                                            // room for 8192 processors
    if (sched_getaffinity(0, sizeof set, set)) return 1;
    const int n = CPU_COUNT_S(sizeof set, set);
    return n < quota ? n : quota;
}

// Into a piece (16-byte aligned) that the link reads next, past the caches: out of the caches of cores that have gone to sleep
// meanwhile it reads slowly. A call with 2 MB of rows, 2 ms after the one before: 250 us when the helpers slept 25 us after they had
// copied, 179 when they stayed awake for 250; past the caches 138, and 125 instead of 160 without the pause.
inline void copy_past_caches(void *to, const void *from, size_t n) {
#if defined(__SSE2__)
    __m128i *d = (__m128i *)to;
    const __m128i *f = (const __m128i *)from;
    for (; n >= 64; n -= 64, d += 4, f += 4) {
        const __m128i a = _mm_loadu_si128(f), b = _mm_loadu_si128(f + 1), c = _mm_loadu_si128(f + 2), e = _mm_loadu_si128(f + 3);
        _mm_stream_si128(d, a);
        _mm_stream_si128(d + 1, b);
        _mm_stream_si128(d + 2, c);
        _mm_stream_si128(d + 3, e);
    }
    memcpy(d, f, n);
    _mm_sfence();                                                // before the part counts as copied
#else
    memcpy(to, from, n);
#endif
}

// A transfer as parts of at most PART bytes in the order of the pieces. Parts below `open` may be taken.
struct Part { void *to; const void *from; size_t n; int piece; };
struct Job {
    bool to_link = false;                                        // the parts go into pieces
    std::vector<Part> parts;
    std::vector<int> left;                                       // per piece: parts in it
    std::vector<std::atomic<int>> done;                          // ... copied
    std::atomic<int> open{0}, next{0}, copied{0};
    explicit Job(size_t pieces) : left(pieces, 0), done(pieces) { for (auto &d : done) d.store(0); }
    bool some() const { return next.load() < open.load(); }
    bool left_over() const { return next.load() < (int)parts.size(); }
    bool worth_waking() const { return some() && next.load() + FRESH < (int)parts.size(); }
    bool take() {
        int i = next.load(std::memory_order_relaxed);
        do if (i >= open.load()) return false;
        while (!next.compare_exchange_weak(i, i + 1));
        const Part &p = parts[(size_t)i];
        if (to_link) copy_past_caches(p.to, p.from, p.n);
        else memcpy(p.to, p.from, p.n);
        done[(size_t)p.piece].fetch_add(1);
        copied.fetch_add(1);
        return true;
    }
    bool ready(int piece) const { return done[(size_t)piece].load() == left[(size_t)piece]; }
};

// Page-locked pieces, and per device the events behind their copies.
struct Set {
    bool held = false;
    uint8_t *base = nullptr;
    cudaEvent_t on_link = nullptr;                               // behind the last piece of a transfer to the device: free once it has left
    std::vector<cudaEvent_t> events[MB_MAX_DEVICES];
    cudaEvent_t *ev = nullptr;                                   // the current device's
    bool prepare() {
        int dev = 0;
        bool ok = !on_link || cudaEventSynchronize(on_link) == cudaSuccess;
        on_link = nullptr;
        ok = ok && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < MB_MAX_DEVICES;
        if (ok && !base && cudaHostAlloc((void **)&base, PIECE * SLOTS, cudaHostAllocPortable) != cudaSuccess) { base = nullptr; ok = false; }
        while (ok && events[dev].size() < (size_t)SLOTS + 1) {
            cudaEvent_t e = nullptr;
            ok = cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
            if (ok) events[dev].push_back(e);
        }
        if (!ok) { cudaGetLastError(); return false; }
        ev = events[dev].data();
        return true;
    }
    void give_back() {
        if (on_link) cudaEventSynchronize(on_link);
        on_link = nullptr;
        for (auto &per : events) { for (cudaEvent_t e : per) cudaEventDestroy(e); per.clear(); }
        if (base) cudaFreeHost(base);
        base = nullptr;
        cudaGetLastError();
    }
};

class Copier {
public:
    std::mutex helped;                                           // held by the transfer that has the helpers

    void user(int d) {
        std::lock_guard<std::mutex> pl(pool_);
        if (users_ == 0) quota_.store(quota_cores(), std::memory_order_relaxed);
        users_ += d;
        if (users_ > 0) return;                                  // (a transfer under way has a user)
        {
            std::lock_guard<std::mutex> lk(mu_);
            leave_ = true;
            wake_.notify_all();
        }
        if (pid_ == getpid()) for (std::thread &t : helpers_) t.join();
        else for (std::thread &t : helpers_) t.detach();         // a fork's child has no such threads
        helpers_.clear();
        leave_ = false;
        RelaxedCapture relaxed;
        for (Set &s : sets_) s.give_back();
    }
    int cores() const { return caller_cores(quota_.load(std::memory_order_relaxed)); }
    // a set of pieces, free again, and helpers for a caller with that many cores; null where there are none
    Set *take(int cores) {
        Set *s = nullptr;
        {
            std::lock_guard<std::mutex> pl(pool_);
            if (helpers_.empty()) pid_ = getpid();
            if (pid_ == getpid()) {
                try {
                    while ((int)helpers_.size() < HELPERS && (int)helpers_.size() + 1 < cores) helpers_.emplace_back([this] { help(); });
                } catch (...) {}                                 // fewer of them
            }
            auto rank = [](const Set &t) { return !t.base ? 0 : t.on_link ? 1 : 2; };
            for (Set &t : sets_) if (!t.held && (!s || rank(t) > rank(*s))) s = &t;
            if (!s) return nullptr;
            s->held = true;
        }
        if (s->prepare()) return s;
        give(s);
        return nullptr;
    }
    void give(Set *s) {
        std::lock_guard<std::mutex> pl(pool_);
        s->held = false;
    }
    // with `helped`, from here on
    void begin(std::shared_ptr<Job> j) {
        std::lock_guard<std::mutex> lk(mu_);
        job_ = std::move(j);
        asked_.fetch_add(1);
        asleep_ = 0;
        wake_.notify_all();
    }
    // parts up to there may be taken (a helper says that it sleeps before it looks for the last time)
    void open(Job &j, int upto) {
        j.open.store(upto);
        if (asleep_.load() == 0) return;
        std::lock_guard<std::mutex> lk(mu_);
        asleep_ = 0;
        wake_.notify_all();
    }
    // the caller's wait for the helpers' parts (a helper looks for a sleeping caller behind each of its parts)
    template <typename F> void await(F ready) {
        if (spin(PATIENCE, ready)) return;
        std::unique_lock<std::mutex> lk(mu_);
        caller_sleeps_ = true;
        while (!ready()) done_.wait(lk);
        caller_sleeps_ = false;
    }
    void end() {
        std::lock_guard<std::mutex> lk(mu_);
        job_ = nullptr;
    }

private:
    void help() {
        sched_param none{};
        sched_setscheduler(0, SCHED_BATCH, &none);               // a woken helper does not take another process's core from it
        unsigned seen = 0;
        for (;;) {
            std::shared_ptr<Job> j;
            {
                std::unique_lock<std::mutex> lk(mu_);
                for (;;) {
                    asleep_++;
                    if (leave_) return;
                    // a transfer that is about to begin, or parts enough
                    if (job_ && ((asked_.load() != seen && job_->open.load() == 0) || job_->worth_waking())) break;
                    wake_.wait(lk);
                }
                asleep_--;
                seen = asked_.load();
                j = job_;
            }
            do
                while (j->take())
                    if (caller_sleeps_.load()) {
                        std::lock_guard<std::mutex> lk(mu_);
                        done_.notify_one();
                    }
            while (spin(j->left_over() ? PATIENCE : LOOK, [&] { return j->some() || asked_.load() != seen; }) && asked_.load() == seen);
        }
    }

    std::mutex mu_;                                              // the helpers' sleep
    std::condition_variable wake_, done_;
    std::atomic<unsigned> asked_{0};                             // transfers so far
    std::atomic<int> asleep_{0};                                 // helpers that nobody has woken yet
    std::atomic<bool> caller_sleeps_{false};
    std::shared_ptr<Job> job_;
    bool leave_ = false;

    std::mutex pool_;                                            // what follows
    Set sets_[SETS];
    int users_ = 0;
    pid_t pid_ = 0;
    std::vector<std::thread> helpers_;
    std::atomic<int> quota_{1};
};
Copier &copier() { static Copier *c = new Copier(); return *c; }  // alive until the process ends

bool pageable(const void *host) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) { cudaGetLastError(); return false; }
    return at.type == cudaMemoryTypeUnregistered;
}
int failed(const char *what, cudaError_t e) {
    cudaGetLastError();
    set_error("%s: %s", what, cudaGetErrorString(e));
    return -1;
}

// The caller's side of a transfer. Whatever happens, it ends with no helper at a part (a helper may still look at the job, which
// lives as long as it is looked at), and with the pieces given back.
struct Transfer {
    Copier &c;
    Set *s;
    const std::shared_ptr<Job> job;
    Job &j;
    std::unique_lock<std::mutex> helped;
    Transfer(Copier &c_, Set *s_, size_t pieces) : c(c_), s(s_), job(std::make_shared<Job>(pieces)), j(*job), helped(c_.helped, std::defer_lock) {}
    ~Transfer() {
        const int taken = j.next.exchange((int)j.parts.size());  // all of them, unless an error came between
        if (helped.owns_lock()) {
            c.end();
            c.await([&] { return j.copied.load() == taken; });
            helped.unlock();
        }
        c.give(s);
    }
    void ask_helpers() { if (helped.try_lock()) c.begin(job); }
    void open(int upto) {
        if (helped.owns_lock()) c.open(j, upto);
        else j.open.store(upto);
    }
    void finish(int piece) {
        while (!j.ready(piece) && j.take()) {}
        c.await([&] { return j.ready(piece); });
    }
};

}  // namespace

void copy_user_made() { copier().user(1); }
void copy_user_gone() { copier().user(-1); }

int copy_in(void *dev, const void *host, size_t bytes, cudaStream_t st) {
    Copier &c = copier();
    RelaxedCapture relaxed;
    const int cores = bytes >= LEAST_IN ? c.cores() : 1;
    Set *s = cores > 1 && pageable(host) ? c.take(cores) : nullptr;
    if (!s) {
        const cudaError_t e = cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
        return e == cudaSuccess ? 0 : failed("copy to the device", e);
    }
    const int n = (int)((bytes + PIECE - 1) / PIECE);
    Transfer t(c, s, (size_t)n);
    Job &j = t.j;
    j.to_link = true;
    for (size_t at = 0; at < bytes; at += PART) {
        const int p = (int)(at / PIECE);
        j.parts.push_back(Part{s->base + (size_t)(p % SLOTS) * PIECE + at % PIECE, (const uint8_t *)host + at, bytes - at < PART ? bytes - at : PART, p});
        j.left[(size_t)p]++;
    }
    t.ask_helpers();
    t.open(n <= SLOTS ? (int)j.parts.size() : SLOTS * PARTS);
    cudaError_t e = cudaSuccess;
    for (int p = 0; p < n && e == cudaSuccess; p++) {
        t.finish(p);
        const size_t at = (size_t)p * PIECE;
        e = cudaMemcpyAsync((uint8_t *)dev + at, s->base + (size_t)(p % SLOTS) * PIECE, bytes - at < PIECE ? bytes - at : PIECE, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(s->ev[p % SLOTS], st);
        // the place of a piece that has left is opened for the piece SLOTS behind it, half the places ahead of need
        const int old = p - SLOTS / 2;
        if (e == cudaSuccess && old >= 0 && old + SLOTS < n) {
            e = cudaEventSynchronize(s->ev[old % SLOTS]);
            const int open = (old + SLOTS + 1) * PARTS;
            if (e == cudaSuccess) t.open(open < (int)j.parts.size() ? open : (int)j.parts.size());
        }
    }
    if (e == cudaSuccess) { s->on_link = s->ev[(n - 1) % SLOTS]; return 0; }
    cudaStreamSynchronize(st);
    return failed("copy to the device", e);
}

int copy_out(const std::vector<CopyOut> &parts, cudaStream_t st) {
    size_t total = 0;
    for (const CopyOut &o : parts) total += o.bytes;
    Copier &c = copier();
    RelaxedCapture relaxed;
    const int cores = total >= LEAST_OUT ? c.cores() : 1;
    bool page = cores > 1;
    for (const CopyOut &o : parts) page = page && (!o.bytes || pageable(o.host));
    Set *s = page ? c.take(cores) : nullptr;
    if (!s) {
        for (const CopyOut &o : parts) {
            const cudaError_t e = o.bytes ? cudaMemcpyAsync(o.host, o.dev, o.bytes, cudaMemcpyDeviceToHost, st) : cudaSuccess;
            if (e != cudaSuccess) return failed("copy to the host", e);
        }
        return 0;
    }
    // pieces end with their part of the caller's memory
    struct Piece { const void *dev; size_t n; };
    std::vector<Piece> pieces;
    for (const CopyOut &o : parts)
        for (size_t at = 0; at < o.bytes; at += PIECE) pieces.push_back(Piece{(const uint8_t *)o.dev + at, o.bytes - at < PIECE ? o.bytes - at : PIECE});
    const int n = (int)pieces.size();
    Transfer t(c, s, (size_t)n);
    Job &j = t.j;
    int p = 0;
    for (const CopyOut &o : parts)
        for (size_t at = 0; at < o.bytes; at += PIECE, p++)
            for (size_t in = 0; in < pieces[(size_t)p].n; in += PART, j.left[(size_t)p]++)
                j.parts.push_back(Part{(uint8_t *)o.host + at + in, s->base + (size_t)(p % SLOTS) * PIECE + in, pieces[(size_t)p].n - in < PART ? pieces[(size_t)p].n - in : PART, p});
    int asked = 0, open = 0;
    cudaError_t e = cudaEventRecord(s->ev[SLOTS], st);
    for (int q = 0; q < n && e == cudaSuccess; q++) {
        for (; asked < n && asked < q + SLOTS && e == cudaSuccess; asked++) {
            if (asked >= SLOTS) t.finish(asked - SLOTS);
            e = cudaMemcpyAsync(s->base + (size_t)(asked % SLOTS) * PIECE, pieces[(size_t)asked].dev, pieces[(size_t)asked].n, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(s->ev[asked % SLOTS], st);
        }
        if (e == cudaSuccess && q == 0) {
            // what came before is done: the helpers wake up while the first piece is on the link (20 us of a call that found them
            // asleep)
            e = cudaEventSynchronize(s->ev[SLOTS]);
            t.ask_helpers();
        }
        if (e == cudaSuccess) e = cudaEventSynchronize(s->ev[q % SLOTS]);
        open += j.left[(size_t)q];
        if (e == cudaSuccess) t.open(open);
    }
    for (int q = 0; q < n && e == cudaSuccess; q++) t.finish(q);
    if (e == cudaSuccess) return 0;
    cudaStreamSynchronize(st);
    return failed("copy to the host", e);
}

}  // namespace mb
