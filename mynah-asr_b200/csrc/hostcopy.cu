// Copies between the device and pageable host memory, by way of page-locked pieces that several threads fill or empty.
//
// The driver copies pageable memory through a buffer of its own with one thread: 3 MB in 200 us, 24 MB in 1.2 to 1.4 ms, either
// way, where the link needs 55 us and 430 (page-locked memory). One core's memcpy is the limit (18 GB/s). Here the caller and up
// to three helpers copy parts of pieces of 512 KB, and a piece is on the link while the next ones are being filled.
//
// One transfer at a time has the pieces: another thread's, meanwhile, takes the driver's way, and so do small and page-locked
// ones (all that is ever recorded into a graph here is small) and those of a caller that has no second core for a helper. Nothing
// waits for a helper that has not taken a part yet: without helpers (none could be started, a forked child) the caller copies all of it.
#include "hostcopy.h"

#include <sched.h>
#include <stdio.h>
#include <string.h>
#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <thread>

namespace mb {
namespace {

constexpr size_t PIECE = 512 << 10, PART = 128 << 10;
constexpr int SLOTS = 4;                                         // page-locked pieces: 2 MB (page-locking takes 1 ms per MB, once)
constexpr int HELPERS = 3;
// Below this the driver's way is as fast: 0.75 MB take 62 us in and 77 out there, 40 to 50 by way of the pieces with the helpers
// still asleep.
constexpr size_t LEAST = 512 << 10;
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

// A transfer as parts of at most PART bytes in the order of the pieces. Parts below `open` may be taken.
struct Part { void *to; const void *from; size_t n; int piece; };
struct Job {
    std::vector<Part> parts;
    std::vector<int> left;                                       // per piece: parts in it
    std::vector<std::atomic<int>> done;                          // ... copied
    std::atomic<int> open{0}, next{0};
    explicit Job(size_t pieces) : left(pieces, 0), done(pieces) { for (auto &d : done) d.store(0, std::memory_order_relaxed); }
    bool take() {
        int i = next.load(std::memory_order_relaxed);
        do if (i >= open.load(std::memory_order_acquire)) return false;
        while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
        const Part &p = parts[(size_t)i];
        memcpy(p.to, p.from, p.n);
        done[(size_t)p.piece].fetch_add(1, std::memory_order_release);
        return true;
    }
    bool ready(int piece) const { return done[(size_t)piece].load(std::memory_order_acquire) == left[(size_t)piece]; }
};

class Copier {
public:
    std::mutex busy;                                             // held by the transfer that has the pieces

    void user(int d) {
        std::lock_guard<std::mutex> b(busy);                     // no transfer under way
        if (users_ == 0) quota_.store(quota_cores(), std::memory_order_relaxed);
        users_ += d;
        if (users_ > 0) return;
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
        if (on_link_) cudaEventSynchronize(on_link_);
        on_link_ = nullptr;
        for (auto &per : events_) { for (cudaEvent_t e : per) cudaEventDestroy(e); per.clear(); }
        if (base_) cudaFreeHost(base_);
        base_ = nullptr;
        cudaGetLastError();
    }
    // the last piece of a transfer to the device, still on the link: the pieces are free once it has left
    void on_link(cudaEvent_t e) { on_link_ = e; }
    int cores() const { return caller_cores(quota_.load(std::memory_order_relaxed)); }
    // with `busy` held: the pieces, free again, the helpers for a caller with that many cores and the current device's events;
    // null where there are none
    uint8_t *pieces(int cores, cudaEvent_t **events) {
        if (on_link_ && cudaEventSynchronize(on_link_) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        on_link_ = nullptr;
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MB_MAX_DEVICES) { cudaGetLastError(); return nullptr; }
        if (!base_ && cudaHostAlloc((void **)&base_, PIECE * SLOTS, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); base_ = nullptr; return nullptr; }
        std::vector<cudaEvent_t> &per = events_[dev];
        while (per.size() < (size_t)SLOTS) {
            cudaEvent_t e = nullptr;
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return nullptr; }
            per.push_back(e);
        }
        if (helpers_.empty()) pid_ = getpid();
        if (pid_ == getpid()) {
            try {
                while ((int)helpers_.size() < HELPERS && (int)helpers_.size() + 1 < cores) helpers_.emplace_back([this] { help(); });
            } catch (...) {}                                     // fewer of them
        }
        *events = per.data();
        return base_;
    }
    void begin(Job *j) {
        std::lock_guard<std::mutex> lk(mu_);
        job_ = j;
        asked_.fetch_add(1, std::memory_order_release);
        wake_.notify_all();
    }
    // no helper looks at the job any more
    void end() {
        std::unique_lock<std::mutex> lk(mu_);
        job_ = nullptr;
        if (pid_ == getpid()) idle_.wait(lk, [this] { return inside_ == 0; });
    }

private:
    void help() {
        unsigned seen = 0;
        for (;;) {
            // transfers often come in pairs (rows in, result out): look out for the next one for 100 us before going to sleep
            for (int i = 0; i < 2000 && asked_.load(std::memory_order_acquire) == seen; i++) pause();
            Job *j = nullptr;
            {
                std::unique_lock<std::mutex> lk(mu_);
                wake_.wait(lk, [&] { return leave_ || asked_.load(std::memory_order_relaxed) != seen; });
                if (leave_) return;
                seen = asked_.load(std::memory_order_relaxed);
                j = job_;
                if (j) inside_++;
            }
            if (!j) continue;
            while (j->next.load(std::memory_order_relaxed) < (int)j->parts.size())
                if (!j->take()) pause();
            std::lock_guard<std::mutex> lk(mu_);
            if (--inside_ == 0) idle_.notify_all();
        }
    }
    static void pause() { for (int i = 0; i < 8; i++) cpu_relax(); }

    std::mutex mu_;
    std::condition_variable wake_, idle_;
    std::atomic<unsigned> asked_{0};
    std::atomic<int> quota_{1};
    Job *job_ = nullptr;
    int inside_ = 0, users_ = 0;
    bool leave_ = false;
    pid_t pid_ = 0;
    std::vector<std::thread> helpers_;
    uint8_t *base_ = nullptr;
    cudaEvent_t on_link_ = nullptr;
    std::vector<cudaEvent_t> events_[MB_MAX_DEVICES];
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

// The caller's side of a transfer. Whatever happens, it ends with no helper in the job, and with no piece on the link.
struct Transfer {
    Copier &c;
    Job &j;
    cudaStream_t st;
    cudaEvent_t *ev;
    int used = 0;                                                // events recorded so far
    Transfer(Copier &c_, Job &j_, cudaStream_t s, cudaEvent_t *e) : c(c_), j(j_), st(s), ev(e) { c.begin(&j); }
    ~Transfer() {
        j.next.store((int)j.parts.size(), std::memory_order_relaxed);       // (nothing is left unless an error came between)
        c.end();
    }
    void finish(int piece) { while (!j.ready(piece)) if (!j.take()) cpu_relax(); }
};

}  // namespace

void copy_user_made() { copier().user(1); }
void copy_user_gone() { copier().user(-1); }

int copy_in(void *dev, const void *host, size_t bytes, cudaStream_t st) {
    Copier &c = copier();
    std::unique_lock<std::mutex> lk(c.busy, std::defer_lock);
    cudaEvent_t *ev = nullptr;
    uint8_t *base = nullptr;
    RelaxedCapture relaxed;
    const int cores = bytes >= LEAST ? c.cores() : 1;
    if (cores > 1 && pageable(host) && lk.try_lock()) base = c.pieces(cores, &ev);
    if (!base) {
        if (lk.owns_lock()) lk.unlock();
        const cudaError_t e = cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
        return e == cudaSuccess ? 0 : failed("copy to the device", e);
    }
    const int n = (int)((bytes + PIECE - 1) / PIECE);
    Job j((size_t)n);
    for (size_t at = 0; at < bytes; at += PART) {
        const int p = (int)(at / PIECE);
        j.parts.push_back(Part{base + (size_t)(p % SLOTS) * PIECE + at % PIECE, (const uint8_t *)host + at, bytes - at < PART ? bytes - at : PART, p});
        j.left[(size_t)p]++;
    }
    cudaError_t e = cudaSuccess;
    {
        Transfer t(c, j, st, ev);
        j.open.store(n <= SLOTS ? (int)j.parts.size() : SLOTS * PARTS, std::memory_order_release);
        for (int p = 0; p < n && e == cudaSuccess; p++) {
            t.finish(p);
            const size_t at = (size_t)p * PIECE;
            e = cudaMemcpyAsync((uint8_t *)dev + at, base + (size_t)(p % SLOTS) * PIECE, bytes - at < PIECE ? bytes - at : PIECE, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(ev[p % SLOTS], st);
            // the place of a piece that has left is opened for the piece SLOTS behind it, half the places ahead of need
            const int old = p - SLOTS / 2;
            if (e == cudaSuccess && old >= 0 && old + SLOTS < n) {
                e = cudaEventSynchronize(ev[old % SLOTS]);
                const int open = (old + SLOTS + 1) * PARTS;
                if (e == cudaSuccess) j.open.store(open < (int)j.parts.size() ? open : (int)j.parts.size(), std::memory_order_release);
            }
        }
    }
    if (e == cudaSuccess) { c.on_link(ev[(n - 1) % SLOTS]); return 0; }
    cudaStreamSynchronize(st);
    return failed("copy to the device", e);
}

int copy_out(const std::vector<CopyOut> &parts, cudaStream_t st) {
    size_t total = 0;
    bool page = true;
    for (const CopyOut &o : parts) total += o.bytes;
    Copier &c = copier();
    std::unique_lock<std::mutex> lk(c.busy, std::defer_lock);
    cudaEvent_t *ev = nullptr;
    uint8_t *base = nullptr;
    RelaxedCapture relaxed;
    const int cores = total >= LEAST ? c.cores() : 1;
    if (cores > 1) {
        for (const CopyOut &o : parts) page = page && (!o.bytes || pageable(o.host));
        if (page && lk.try_lock()) base = c.pieces(cores, &ev);
    }
    if (!base) {
        if (lk.owns_lock()) lk.unlock();
        for (const CopyOut &o : parts) {
            const cudaError_t e = o.bytes ? cudaMemcpyAsync(o.host, o.dev, o.bytes, cudaMemcpyDeviceToHost, st) : cudaSuccess;
            if (e != cudaSuccess) return failed("copy to the host", e);
        }
        return 0;
    }
    // pieces end with their part of the caller's memory
    struct Piece { const void *dev; size_t n; int parts; };
    std::vector<Piece> pieces;
    for (const CopyOut &o : parts)
        for (size_t at = 0; at < o.bytes; at += PIECE) pieces.push_back(Piece{(const uint8_t *)o.dev + at, o.bytes - at < PIECE ? o.bytes - at : PIECE, 0});
    const int n = (int)pieces.size();
    Job j((size_t)n);
    int p = 0;
    for (const CopyOut &o : parts)
        for (size_t at = 0; at < o.bytes; at += PIECE, p++)
            for (size_t in = 0; in < pieces[(size_t)p].n; in += PART, j.left[(size_t)p]++)
                j.parts.push_back(Part{(uint8_t *)o.host + at + in, base + (size_t)(p % SLOTS) * PIECE + in, pieces[(size_t)p].n - in < PART ? pieces[(size_t)p].n - in : PART, p});
    cudaError_t e = cudaSuccess;
    {
        Transfer t(c, j, st, ev);
        int asked = 0, open = 0;
        for (int q = 0; q < n && e == cudaSuccess; q++) {
            for (; asked < n && asked < q + SLOTS && e == cudaSuccess; asked++) {
                if (asked >= SLOTS) t.finish(asked - SLOTS);
                e = cudaMemcpyAsync(base + (size_t)(asked % SLOTS) * PIECE, pieces[(size_t)asked].dev, pieces[(size_t)asked].n, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[asked % SLOTS], st);
            }
            if (e == cudaSuccess) e = cudaEventSynchronize(ev[q % SLOTS]);
            open += j.left[(size_t)q];
            if (e == cudaSuccess) j.open.store(open, std::memory_order_release);
        }
        for (int q = 0; q < n && e == cudaSuccess; q++) t.finish(q);
    }
    if (e == cudaSuccess) return 0;
    cudaStreamSynchronize(st);
    return failed("copy to the host", e);
}

}  // namespace mb
