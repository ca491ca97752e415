// Host copies through pinned staging memory.
//
// A cudaMemcpy on pageable memory moves 7 GB/s here: the driver stages it through
// one thread, which also takes the page faults of freshly allocated result arrays
// (21 MB of a 525,825-point state: 2.9 ms).  Here the DMA runs from and to two
// pinned halves in turn while several threads copy the other half: 1.8 ms for that
// state (what is left is its page faults), 0.4 in place of 1.1 ms for two arrays
// of it in; halves of 1 to 8 MB and eight threads were no faster.  Where the system
// refuses pinned memory or events, the copies are plain ones.
#include <condition_variable>
#include <mutex>
#include <thread>

#include "fs_internal.h"

namespace fsb {

namespace {

constexpr size_t kHalf = size_t(2) << 20;   // bytes per pinned half
constexpr int kStages = 4;                  // staging pieces kept at most
constexpr int kCopyThreads = 4;             // the caller's among them
constexpr size_t kShare = size_t(128) << 10;  // least bytes worth a thread
// Staging memory costs 4.5 ms: 3.8 to allocate 4 MB of it, 0.7 to give it back.  It
// saves 0.28 ms per MB copied out (to fresh pages: 7.2 -> 2.5 ms for 16 MB), a tenth
// of that in, and 10 us of a short call.  So it is allocated once copies would have
// saved about as much, since the first HostStage that lives: an object of one call,
// which took 0.7 ms with its creation at 2,145 points and 5.4 with staging memory of
// its own, does without; the two-stream state of 525,825 points stages at once.
constexpr size_t kWorth = size_t(16) << 20;      // bytes out, or 8 times as many in
constexpr size_t kWorthLeast = size_t(32) << 10;  // of any call

// Threads that copy pieces of memory for whoever asks; they live while a
// HostStage does.  Fewer threads than asked for (none, where the system refuses
// them) only make the caller copy more.
class CopyThreads {
   public:
    ~CopyThreads() { stop(); }
    void copy(char* dst, const char* src, size_t bytes) {
        const size_t parts = std::min<size_t>(kCopyThreads, std::max<size_t>(1, bytes / kShare));
        if (parts == 1) {
            std::memcpy(dst, src, bytes);
            return;
        }
        const size_t per = (bytes / parts + 4095) & ~size_t(4095);
        Piece piece[kCopyThreads];
        int left = 0;
        {
            std::lock_guard<std::mutex> lk(mu_);
            start();
            for (size_t k = 1; k < parts && k * per < bytes; ++k) {
                piece[k] = {dst + k * per, src + k * per, std::min(per, bytes - k * per), &left, nullptr};
                (last_ ? last_->next : first_) = &piece[k];
                last_ = &piece[k];
                ++left;
            }
        }
        cv_.notify_all();
        std::memcpy(dst, src, std::min(per, bytes));
        std::unique_lock<std::mutex> lk(mu_);
        while (left > 0) {
            if (first_) run_one(lk);
            else done_.wait(lk);
        }
    }
    void stop() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stopping_ = true;
        }
        cv_.notify_all();
        for (auto& t : threads_) t.join();
        threads_.clear();
        stopping_ = false;
    }

   private:
    struct Piece {
        char* dst;
        const char* src;
        size_t bytes;
        int* left;
        Piece* next;
    };
    void start() {
        while ((int)threads_.size() < kCopyThreads - 1) {
            try {
                threads_.emplace_back([this] { work(); });
            } catch (...) {
                return;
            }
        }
    }
    void run_one(std::unique_lock<std::mutex>& lk) {
        const Piece p = *first_;
        first_ = p.next;
        if (!first_) last_ = nullptr;
        lk.unlock();
        std::memcpy(p.dst, p.src, p.bytes);
        lk.lock();
        if (--*p.left == 0) done_.notify_all();
    }
    void work() {
        std::unique_lock<std::mutex> lk(mu_);
        for (;;) {
            cv_.wait(lk, [&] { return stopping_ || first_; });
            if (!first_) return;
            run_one(lk);
        }
    }
    std::mutex mu_;
    std::condition_variable cv_, done_;
    Piece *first_ = nullptr, *last_ = nullptr;  // pieces that nobody has taken, in their callers' frames
    std::vector<std::thread> threads_;
    bool stopping_ = false;
};

struct Piece {
    char* half[2] = {nullptr, nullptr};
};

// What the HostStages share.
struct Shared {
    std::mutex mu;
    std::condition_variable cv;
    int users = 0, pieces = 0;
    size_t worth = 0;  // of the copies without staging memory
    std::vector<Piece> free;
    CopyThreads threads;
};
Shared& shared() {
    static Shared* s = new Shared;  // not destroyed at exit: stages may outlive statics
    return *s;
}

// One staging piece for the length of a copy, or none where it is not worth one yet
// or the system refuses pinned memory or events.  No DMA uses it any more when it
// goes back, whatever happened.
class Hold {
   public:
    explicit Hold(size_t worth) {
        Shared& s = shared();
        {
            std::unique_lock<std::mutex> lk(s.mu);
            if (s.pieces == 0) {
                s.worth += std::max(worth, kWorthLeast);
                if (s.worth < kWorth) return;
                s.worth = 0;  // (if it is refused, not asked for at every call)
            }
            held_ = true;
            s.cv.wait(lk, [&] { return !s.free.empty() || s.pieces < kStages; });
            if (!s.free.empty()) {
                p_ = s.free.back();
                s.free.pop_back();
            } else {
                ++s.pieces;
            }
        }
        if (!p_.half[0]) {
            void* m = nullptr;
            if (cudaHostAlloc(&m, 2 * kHalf, cudaHostAllocPortable) == cudaSuccess) {
                p_.half[0] = static_cast<char*>(m);
                p_.half[1] = p_.half[0] + kHalf;
            } else {
                (void)cudaGetLastError();
            }
        }
        ok_ = p_.half[0] != nullptr;
        for (auto& e : ev_)
            if (ok_ && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                (void)cudaGetLastError();
                e = nullptr;
                ok_ = false;
            }
    }
    ~Hold() { end(); }
    bool ok() const { return ok_; }
    char* half(int k) const { return p_.half[k]; }
    // Copies of half k follow on `st`, until its record().
    void begin(int k, cudaStream_t st) {
        st_ = st;
        open_[k] = true;
    }
    void record(int k) {
        FS_CUDA(cudaEventRecord(ev_[k], st_));
        busy_[k] = true;
        open_[k] = false;
    }
    void wait(int k) {
        if (!busy_[k]) return;
        FS_CUDA(cudaEventSynchronize(ev_[k]));
        busy_[k] = false;
    }

   private:
    void end() {
        if (!held_) return;
        if (open_[0] || open_[1]) (void)cudaStreamSynchronize(st_);  // copies that no event follows
        for (int k = 0; k < 2; ++k) {
            if (busy_[k]) (void)cudaEventSynchronize(ev_[k]);
            if (ev_[k]) cudaEventDestroy(ev_[k]);
        }
        give_back();
    }
    void give_back() {
        Shared& s = shared();
        {
            std::lock_guard<std::mutex> lk(s.mu);
            if (p_.half[0]) s.free.push_back(p_);
            else --s.pieces;
        }
        s.cv.notify_one();
    }
    Piece p_;
    cudaEvent_t ev_[2] = {nullptr, nullptr};
    cudaStream_t st_ = nullptr;
    bool held_ = false, ok_ = false, busy_[2] = {false, false}, open_[2] = {false, false};
};

// The copies cut into pieces and gathered into loads of at most one half.
struct Chunk {
    char* dst;
    const char* src;
    size_t bytes, at;  // place in the half
};
std::vector<std::vector<Chunk>> loads_of(const std::vector<HostCopy>& copies) {
    std::vector<std::vector<Chunk>> v;
    size_t used = kHalf;
    for (const HostCopy& c : copies)
        for (size_t o = 0; o < c.bytes;) {
            if (used >= kHalf) {
                v.emplace_back();
                used = 0;
            }
            const size_t b = std::min(kHalf - used, c.bytes - o);
            v.back().push_back({static_cast<char*>(c.dst) + o, static_cast<const char*>(c.src) + o, b, used});
            used = (used + b + 255) & ~size_t(255);
            o += b;
        }
    return v;
}

size_t total(const std::vector<HostCopy>& copies) {
    size_t b = 0;
    for (const HostCopy& c : copies) b += c.bytes;
    return b;
}

}  // namespace

HostStage::HostStage() {
    Shared& s = shared();
    std::lock_guard<std::mutex> lk(s.mu);
    ++s.users;
}

HostStage::~HostStage() {
    Shared& s = shared();
    std::vector<Piece> go;
    {
        std::lock_guard<std::mutex> lk(s.mu);
        if (--s.users > 0) return;
        s.worth = 0;
        go.swap(s.free);
        s.pieces -= (int)go.size();
        s.threads.stop();
    }
    for (const Piece& p : go) cudaFreeHost(p.half[0]);
}

void HostStage::to_host(const std::vector<HostCopy>& copies, cudaStream_t st) {
    const std::vector<std::vector<Chunk>> v = loads_of(copies);
    if (v.empty()) {
        FS_CUDA(cudaStreamSynchronize(st));
        return;
    }
    Hold h(total(copies));
    if (!h.ok()) {
        for (const HostCopy& c : copies) FS_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, st));
        FS_CUDA(cudaStreamSynchronize(st));
        return;
    }
    auto issue = [&](size_t k) {
        h.begin(k & 1, st);
        for (const Chunk& c : v[k])
            FS_CUDA(cudaMemcpyAsync(h.half(k & 1) + c.at, c.src, c.bytes, cudaMemcpyDeviceToHost, st));
        h.record(k & 1);
    };
    for (size_t k = 0; k < std::min<size_t>(2, v.size()); ++k) issue(k);
    for (size_t k = 0; k < v.size(); ++k) {
        h.wait(k & 1);
        for (const Chunk& c : v[k]) shared().threads.copy(c.dst, h.half(k & 1) + c.at, c.bytes);
        if (k + 2 < v.size()) issue(k + 2);
    }
}

void HostStage::to_device(const std::vector<HostCopy>& copies, cudaStream_t st) {
    const std::vector<std::vector<Chunk>> v = loads_of(copies);
    if (v.empty()) return;
    Hold h(total(copies) / 8);
    if (!h.ok()) {
        for (const HostCopy& c : copies) FS_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyHostToDevice, st));
        return;
    }
    for (size_t k = 0; k < v.size(); ++k) {
        h.wait(k & 1);
        h.begin(k & 1, st);
        for (const Chunk& c : v[k]) {
            shared().threads.copy(h.half(k & 1) + c.at, c.src, c.bytes);
            FS_CUDA(cudaMemcpyAsync(c.dst, h.half(k & 1) + c.at, c.bytes, cudaMemcpyHostToDevice, st));
        }
        h.record(k & 1);
    }
}

}  // namespace fsb
