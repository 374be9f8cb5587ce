// hostcopy.cu — large copies between the caller's (pageable) memory and the device.
//
// A pageable cudaMemcpyAsync moves its bytes through the driver's pinned buffer
// with one host thread.  Into memory that has not been touched yet (a new
// array) that is slow, since every page is zeroed on the way: 1 MB 494 us, 6 MB
// 2.9 ms, 36 MB 17 ms (82 us, 0.4 and 2.1 ms into used memory).  Here the copy
// engine fills a ring of pinned buffers which the caller, and from HELP_MIN on a
// few threads, empty: 329 us, 1.0 and 5.2 ms (76 us, 0.3 and 1.2 ms).  Waking the
// threads costs about 100 us, so less is left to the caller.  Uploads read used
// memory: 36 MB 1.9 -> 1.35 ms, 12 MB no gain, so only those of UP_MIN go this way.
//
// What it keeps is shared by all contexts of the process: THREADS helpers, and
// at most LEASES rings, one per copy in progress (a copy that finds none free
// goes the plain way).  The last context to close gives all of it back.
#include "hostcopy.cuh"

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace rcmvs {
namespace {

constexpr size_t SLOT = 1 << 20;
constexpr int SLOTS = 6, LEASES = 4;
constexpr unsigned THREADS = 3;
constexpr size_t DOWN_MIN = 256 << 10, UP_MIN = 24 << 20, HELP_MIN = 3 << 20;

struct Task {
    void* to;
    const void* from;
    size_t n;
    std::atomic<int>* done;
};

// Helper threads with one queue; a waiting caller runs tasks itself.
class Helpers {
  public:
    void start() {
        std::lock_guard<std::mutex> l(m_);
        if (!threads_.empty()) return;
        stop_ = false;
        pid_ = getpid();
        const unsigned cores = std::thread::hardware_concurrency();
        const unsigned n = std::min(THREADS, cores > 1 ? cores - 1 : 0u);
        try {
            while (threads_.size() < n) threads_.emplace_back([this] { loop(); });
        } catch (const std::exception&) {  // no thread or no memory: fewer, or none, and the callers do the work
        }
    }
    // Of this process: a forked child has the objects but not the threads.
    bool mine() const { return threads_.empty() || pid_ == getpid(); }
    void stop() {
        if (!mine()) {
            for (std::thread& t : threads_) t.detach();
            threads_.clear();
            return;
        }
        {
            std::lock_guard<std::mutex> l(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (std::thread& t : threads_) t.join();
        threads_.clear();
    }
    void submit(const Task& t) {
        try {
            std::lock_guard<std::mutex> l(m_);
            q_.push_back(t);
        } catch (const std::bad_alloc&) {
            return run(t);
        }
        cv_.notify_one();
    }
    static void run(const Task& t) {
        std::memcpy(t.to, t.from, t.n);
        t.done->store(1, std::memory_order_release);
    }
    bool help() {
        Task t;
        {
            std::lock_guard<std::mutex> l(m_);
            if (q_.empty()) return false;
            t = q_.front();
            q_.pop_front();
        }
        run(t);
        return true;
    }

  private:
    void loop() {
        std::unique_lock<std::mutex> l(m_);
        for (;;) {
            cv_.wait(l, [this] { return stop_ || !q_.empty(); });
            if (q_.empty()) return;  // stop, with nothing left to do
            const Task t = q_.front();
            q_.pop_front();
            l.unlock();
            run(t);
            l.lock();
        }
    }
    std::mutex m_;
    std::condition_variable cv_;
    std::deque<Task> q_;
    std::vector<std::thread> threads_;
    bool stop_ = false;
    pid_t pid_ = 0;
};

struct Ring {
    int device = 0;
    char* mem = nullptr;
    cudaEvent_t ev[SLOTS] = {};
    bool queued[SLOTS] = {};  // a copy engine's work on the slot may be in flight
    bool busy = false;
};

struct Service {
    Service() { rings.reserve(LEASES); }
    std::mutex m;
    int users = 0;
    std::vector<Ring*> rings;
    Helpers helpers;
};
// never destroyed: threads may outlive static destruction at exit.  Made by the
// first context; only that may throw.
Service& service() {
    static Service* s = new Service;
    return *s;
}

void free_ring(Ring* r) {
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(r->device);
    for (int i = 0; i < SLOTS; ++i)
        if (r->ev[i]) {
            if (r->queued[i]) cudaEventSynchronize(r->ev[i]);
            cudaEventDestroy(r->ev[i]);
        }
    if (r->mem) cudaFreeHost(r->mem);
    delete r;
    cudaSetDevice(cur);
}

// A free ring of the current device, or null.
Ring* take_ring() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    Service& s = service();
    std::lock_guard<std::mutex> l(s.m);
    if (s.users == 0 || !s.helpers.mine()) return nullptr;
    for (Ring* r : s.rings)
        if (!r->busy && r->device == dev) {
            r->busy = true;
            return r;
        }
    if (s.rings.size() >= LEASES) {
        // make room with an idle ring of another device
        auto it = std::find_if(s.rings.begin(), s.rings.end(), [](Ring* r) { return !r->busy; });
        if (it == s.rings.end()) return nullptr;
        free_ring(*it);
        s.rings.erase(it);
    }
    Ring* r = new (std::nothrow) Ring;
    if (!r) return nullptr;
    r->device = dev;
    bool ok = cudaHostAlloc((void**)&r->mem, SLOT * SLOTS, cudaHostAllocDefault) == cudaSuccess;
    for (int i = 0; i < SLOTS && ok; ++i) ok = cudaEventCreateWithFlags(&r->ev[i], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();  // the plain way serves
        free_ring(r);
        return nullptr;
    }
    s.helpers.start();
    r->busy = true;
    s.rings.push_back(r);
    return r;
}

void give_ring(Ring* r) {
    Service& s = service();
    std::lock_guard<std::mutex> l(s.m);
    r->busy = false;
}

// Whether a copy goes through the ring: enough bytes, pageable, and no capture
// in progress (a capture records plain copies only).
bool through_ring(const void* host, size_t n, cudaStream_t st, bool up) {
    if (n < (up ? UP_MIN : DOWN_MIN)) return false;
    cudaStreamCaptureStatus cap;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// done: one zero for each piece.
cudaError_t ring_copy(Ring* r, char* dev, char* host, size_t bytes, std::atomic<int>* done, int n, cudaStream_t st,
                      bool up) {
    Helpers& h = service().helpers;
    auto size = [&](int k) { return std::min(SLOT, bytes - SLOT * k); };
    auto slot = [&](int k) { return r->mem + SLOT * (k % SLOTS); };
    auto hand_over = [&](int k) {  // the host's part of piece k
        char* p = host + SLOT * k;
        const Task t{up ? slot(k) : p, up ? p : slot(k), size(k), &done[k]};
        if (bytes >= HELP_MIN)
            h.submit(t);
        else
            Helpers::run(t);
    };
    auto wait = [&](int k) {
        while (!done[k].load(std::memory_order_acquire))
            if (!h.help()) std::this_thread::yield();
    };
    cudaError_t e = cudaSuccess;
    int given = 0;  // pieces handed over
    int queued = 0;
    for (int k = 0; k < n && e == cudaSuccess; ++k) {
        if (up) {
            // threads fill slots ahead; the copy engine empties them in order
            for (; given < n && given < k + SLOTS; ++given) {
                const int s = given % SLOTS;
                if (r->queued[s]) {
                    if (given > k && cudaEventQuery(r->ev[s]) != cudaSuccess) break;
                    if ((e = cudaEventSynchronize(r->ev[s])) != cudaSuccess) break;
                    r->queued[s] = false;
                }
                hand_over(given);
            }
            if (e != cudaSuccess) break;
            wait(k);
            e = cudaMemcpyAsync(dev + SLOT * k, slot(k), size(k), cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(r->ev[k % SLOTS], st);
            if (e == cudaSuccess) r->queued[k % SLOTS] = true;
        } else {
            // the copy engine fills slots ahead; threads empty them
            for (; queued < n && queued < k + SLOTS; ++queued) {
                const int s = queued % SLOTS;
                if (queued >= SLOTS && !done[queued - SLOTS].load(std::memory_order_acquire)) {
                    if (queued > k) break;
                    wait(queued - SLOTS);
                }
                if (r->queued[s] && (e = cudaEventSynchronize(r->ev[s])) != cudaSuccess) break;
                e = cudaMemcpyAsync(slot(queued), dev + SLOT * queued, size(queued), cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(r->ev[s], st);
                if (e != cudaSuccess) break;
                r->queued[s] = true;
            }
            if (e != cudaSuccess) break;
            if ((e = cudaEventSynchronize(r->ev[k % SLOTS])) != cudaSuccess) break;
            r->queued[k % SLOTS] = false;
            hand_over(k);
            ++given;
        }
    }
    for (int k = 0; k < given; ++k) wait(k);  // no thread keeps the caller's memory
    return e;
}

cudaError_t copy(void* dev, void* host, size_t n, cudaStream_t st, bool up) {
    if (through_ring(host, n, st, up)) {
        const int pieces = (int)((n + SLOT - 1) / SLOT);
        std::unique_ptr<std::atomic<int>[]> done(new (std::nothrow) std::atomic<int>[pieces]());
        if (Ring* r = done ? take_ring() : nullptr) {
            const cudaError_t e = ring_copy(r, (char*)dev, (char*)host, n, done.get(), pieces, st, up);
            give_ring(r);
            return e;
        }
    }
    const cudaError_t e = up ? cudaMemcpyAsync(dev, host, n, cudaMemcpyHostToDevice, st)
                             : cudaMemcpyAsync(host, dev, n, cudaMemcpyDeviceToHost, st);
    return up || e != cudaSuccess ? e : cudaStreamSynchronize(st);
}

}  // namespace

cudaError_t host_upload(void* dev, const void* host, size_t n, cudaStream_t st) {
    return copy(dev, const_cast<void*>(host), n, st, true);
}
cudaError_t host_download(void* host, const void* dev, size_t n, cudaStream_t st) {
    return copy(const_cast<void*>(dev), host, n, st, false);
}

bool host_copy_attach() {
    try {
        Service& s = service();
        std::lock_guard<std::mutex> l(s.m);
        ++s.users;
    } catch (const std::exception&) {
        return false;
    }
    return true;
}

void host_copy_detach() {
    Service& s = service();
    std::lock_guard<std::mutex> l(s.m);
    if (--s.users > 0) return;
    // no context, so no copy in progress
    const bool mine = s.helpers.mine();
    s.helpers.stop();
    if (mine)
        for (Ring* r : s.rings) free_ring(r);
    s.rings.clear();
}

}  // namespace rcmvs
