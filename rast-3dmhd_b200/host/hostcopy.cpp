// hostcopy.cpp - host memory copies by several threads (device transfers of pageable arrays).
#include <omp.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "r3d_host.hpp"

namespace r3db {

namespace {
// Eight blocks to a transfer's chunk.  Half of that puts four threads on the faults of one huge page (an
// adjoint_step of 128x128x128 12.1 ms against 11.8), twice of that leaves half of them idle (13.9).
constexpr size_t kBlock = size_t(1) << 20;
// A transfer's copies follow one another within some 0.3 ms, and a sleeping thread took as long to wake
// (16-core host: upload of five 4.3 MB fields 4.4 ms with threads that sleep at once, 1.3 so).
constexpr std::chrono::microseconds kSpin{1000};

void relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}
}  // namespace

// Not an OpenMP team: that takes the process down when a thread cannot be made, and hangs in a child forked
// after the set-up's parallel loops.
struct CopyTeam::Shared {
    enum State { kReady, kCopying, kAsleep };
    struct Worker {
        std::atomic<int> state{kReady};  // kReady -> kCopying and kAsleep -> kReady: the caller; the others: the thread
        std::thread thread;
    };
    std::vector<Worker> workers;
    size_t made = 0;
    const pid_t owner = getpid();
    std::mutex m;  // kAsleep -> kReady
    std::condition_variable wake;
    std::atomic<bool> stop{false};
    // the copy, set while no worker is at it
    char* dst = nullptr;
    const char* src = nullptr;
    size_t bytes = 0;
    std::atomic<size_t> next{0}, finished{0};

    explicit Shared(size_t n) : workers(n) {}

    bool block() {
        const size_t off = next.fetch_add(kBlock, std::memory_order_relaxed);
        if (off >= bytes) return false;
        std::memcpy(dst + off, src + off, std::min(kBlock, bytes - off));
        return true;
    }
    void work(Worker& w) {
        auto since = std::chrono::steady_clock::now();
        while (!stop.load(std::memory_order_relaxed)) {
            int st = w.state.load(std::memory_order_acquire);
            if (st == kCopying) {
                while (block()) {
                }
                w.state.store(kReady, std::memory_order_relaxed);
                finished.fetch_add(1, std::memory_order_release);
                since = std::chrono::steady_clock::now();
            } else if (std::chrono::steady_clock::now() - since < kSpin) {
                relax();
            } else if (st = kReady; w.state.compare_exchange_strong(st, kAsleep)) {
                std::unique_lock<std::mutex> lock(m);
                wake.wait(lock, [&] { return stop.load() || w.state.load() != kAsleep; });
                since = std::chrono::steady_clock::now();
            }
        }
    }
};

CopyTeam::CopyTeam() : s(nullptr) {
    const int n = std::min({8, omp_get_max_threads(), omp_get_num_procs()});
    s = new Shared((size_t)std::max(n - 1, 0));
    try {
        for (auto& w : s->workers) {
            w.thread = std::thread([this, &w] { s->work(w); });
            ++s->made;
        }
    } catch (const std::exception&) {  // those that could be made
    }
}

CopyTeam::~CopyTeam() {
    if (!mine()) return;  // a forked child has none of the threads: nothing to stop or to free safely
    {
        std::lock_guard<std::mutex> lock(s->m);
        s->stop.store(true);
    }
    s->wake.notify_all();
    for (size_t q = 0; q < s->made; ++q) s->workers[q].thread.join();
    delete s;
}

bool CopyTeam::mine() const { return getpid() == s->owner; }

void CopyTeam::wake() {
    if (!mine()) return;
    bool any = false;
    for (size_t q = 0; q < s->made; ++q)
        if (s->workers[q].state.load() == Shared::kAsleep) {
            std::lock_guard<std::mutex> lock(s->m);
            s->workers[q].state.store(Shared::kReady);
            any = true;
        }
    if (any) s->wake.notify_all();
}

// One thread copies into freshly allocated pages at a few GB/s (it takes their page faults on the
// way), far below the link to the device; eight run at several times that.  Workers join as they come: while
// those asleep wake, the caller copies some blocks.
void CopyTeam::copy(void* dst, const void* src, size_t bytes) {
    if (bytes <= kBlock || s->made == 0 || !mine()) {
        std::memcpy(dst, src, bytes);
        return;
    }
    s->dst = static_cast<char*>(dst);
    s->src = static_cast<const char*>(src);
    s->bytes = bytes;
    s->next.store(0, std::memory_order_relaxed);
    s->finished.store(0, std::memory_order_relaxed);
    wake();
    size_t joined = 0;
    do {
        for (size_t q = 0; q < s->made; ++q) {
            int st = Shared::kReady;
            if (s->workers[q].state.compare_exchange_strong(st, Shared::kCopying)) ++joined;
        }
    } while (s->block());
    while (s->finished.load(std::memory_order_acquire) != joined) relax();
}

std::shared_ptr<CopyTeams> CopyTeams::get() {
    static std::mutex m;
    static std::weak_ptr<CopyTeams> teams;
    std::lock_guard<std::mutex> lock(m);
    auto p = teams.lock();
    if (!p) teams = p = std::make_shared<CopyTeams>();
    return p;
}

CopyTeams::Use::Use(CopyTeams& p) : pool(p) {
    std::lock_guard<std::mutex> lock(pool.m);
    while (!team && !pool.idle.empty()) {
        team = std::move(pool.idle.back());
        pool.idle.pop_back();
        if (!team->mine()) team.reset();
    }
    if (!team) {
        pool.idle.reserve(++pool.made);
        team = std::make_unique<CopyTeam>();
    }
}

CopyTeams::Use::~Use() {
    std::lock_guard<std::mutex> lock(pool.m);
    pool.idle.push_back(std::move(team));
}

}  // namespace r3db
