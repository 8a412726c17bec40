// host_pool.cpp — helper threads for a call's host preparation.
//
// A whole frame's descriptors (tens of thousands of TUs or predictions) cost
// the entry points milliseconds of host time on one thread, several times the
// kernels' time, while the decoder's other cores idle.  The helpers are started
// by the first call large enough to use them, at most kMost of them and at most
// half the cores, and sleep otherwise.  A process forked later has none and
// prepares on its calling threads.
#include "host_pool.h"

#ifdef __SSE2__
#include <emmintrin.h>
#endif
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace av1g {

namespace {

constexpr int kMost = 7;
// Items (TUs, predictions: 20 to 100 ns each) below which waking a helper, some
// 10 us, costs more than it saves.
constexpr long long kAlone = 2048;

struct Task {
    const std::function<void(int)>* fn;
    int n;
    std::atomic<int> next{0};
    int helpers = 0;           // inside it (under the pool's mutex)
    std::exception_ptr error;  // the first one (under the pool's mutex)
};

struct Pool {
    std::mutex mu;
    std::condition_variable work, left;
    std::vector<Task*> open;  // tasks with parts not handed out yet, oldest first
    pid_t pid = getpid();
    int threads = 0, idle = 0;
    bool started = false;

    void run(Task& t) {
        for (;;) {
            const int i = t.next.fetch_add(1, std::memory_order_relaxed);
            if (i >= t.n) return;
            try {
                (*t.fn)(i);
            } catch (...) {
                std::lock_guard<std::mutex> lk(mu);
                if (!t.error) t.error = std::current_exception();
            }
        }
    }

    void helper() {
        std::unique_lock<std::mutex> lk(mu);
        for (;;) {
            idle++;
            while (open.empty()) work.wait(lk);
            idle--;
            Task* t = open.front();
            t->helpers++;
            lk.unlock();
            run(*t);
            lk.lock();
            // nothing of it is left to hand out
            open.erase(std::remove(open.begin(), open.end(), t), open.end());
            if (--t->helpers == 0) left.notify_all();
        }
    }

    // under mu
    void start() {
        started = true;
        const int want = std::min<int>(kMost, (int)std::thread::hardware_concurrency() / 2 - 1);
        for (int k = 0; k < want; k++) {
            try {
                std::thread([this] { helper(); }).detach();
                threads++;
            } catch (...) {  // no thread to be had: the calls do with fewer
                break;
            }
        }
    }
};

Pool& pool() {
    static Pool* p = new Pool;  // never destroyed: helpers wait on it until the process ends
    return *p;
}

}  // namespace

int parallel_parts(long long items, long long grain) {
    return (int)std::max<long long>(1, std::min<long long>(4 * (kMost + 1), items / grain));
}

void parallel_for(int n, long long items, const std::function<void(int)>& fn) {
    if (n <= 0) return;
    Pool& P = pool();
    if (n == 1 || items < kAlone || P.pid != getpid()) {
        for (int i = 0; i < n; i++) fn(i);
        return;
    }
    Task t{&fn, n};
    int wake;
    {
        std::lock_guard<std::mutex> lk(P.mu);
        if (!P.started) P.start();
        P.open.push_back(&t);
        wake = std::min(n - 1, P.threads);
        if (P.idle) wake = std::min(wake, P.idle);
    }
    // no more than there is work for: calls on other threads share the helpers
    for (int k = 0; k < wake; k++) P.work.notify_one();
    P.run(t);
    std::unique_lock<std::mutex> lk(P.mu);
    P.open.erase(std::remove(P.open.begin(), P.open.end(), &t), P.open.end());
    while (t.helpers > 0) P.left.wait(lk);
    if (t.error) std::rethrow_exception(t.error);
}

void write_back(void* p, size_t n) {
#ifdef __SSE2__
    constexpr uintptr_t kLine = 64;
    const uintptr_t a = ((uintptr_t)p + kLine - 1) & ~(kLine - 1), b = ((uintptr_t)p + n) & ~(kLine - 1);
    for (uintptr_t q = a; q < b; q += 16) {
        __m128i* w = reinterpret_cast<__m128i*>(q);
        _mm_stream_si128(w, _mm_load_si128(w));
    }
    _mm_sfence();
#else
    (void)p, (void)n;
#endif
}

}  // namespace av1g
