// Host copies (multi_species_b200/csrc/fs_stage.cpp) against a stand-in for the CUDA
// calls they make: asynchronous copies of pinned memory run when their event or
// stream is waited for, copies of pageable memory at once, and any call can be made
// to fail.  Prints what went wrong; exit code 0 if nothing did.
#include "../multi_species_b200/csrc/fs_stage.cpp"

#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>

namespace {
struct Copy {
    char* dst;
    const char* src;
    size_t bytes;
    long long at;
};
std::deque<Copy> queue;          // one stream
std::map<char*, size_t> pinned;
std::map<void*, long long> events;
long long now = 0;
int copies = 0, records = 0, pins = 0, threads = 0, bad = 0;
int fail_copy = -1, fail_record = -1;
bool fail_pin = false, fail_event = false, fail_thread = false;
const cudaStream_t kStream = reinterpret_cast<cudaStream_t>(8);

void expect(bool ok, const char* what) {
    if (ok) return;
    std::printf("%s\n", what);
    ++bad;
}
bool is_pinned(const void* p) {
    const char* c = static_cast<const char*>(p);
    for (auto& m : pinned)
        if (c >= m.first && c < m.first + m.second) return true;
    return false;
}
void run_until(long long t) {
    while (!queue.empty() && queue.front().at <= t) {
        std::memcpy(queue.front().dst, queue.front().src, queue.front().bytes);
        queue.pop_front();
    }
}
}  // namespace

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    ++pins;
    if (fail_pin) return cudaErrorMemoryAllocation;
    *p = std::malloc(bytes);
    pinned[static_cast<char*>(*p)] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    char* a = static_cast<char*>(p);
    for (const Copy& c : queue)
        expect(!(c.dst >= a && c.dst < a + pinned[a]) && !(c.src >= a && c.src < a + pinned[a]),
               "staging memory given back under a copy");
    pinned.erase(a);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    if (fail_event) return cudaErrorMemoryAllocation;
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    events.erase(e);
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    expect(st == kStream, "event on another stream");
    if (records++ == fail_record) return cudaErrorUnknown;
    events[e] = now;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    run_until(events[e]);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    expect(st == kStream, "wait for another stream");
    run_until(now);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t st) {
    expect(st == kStream, "copy on another stream");
    if (copies++ == fail_copy) return cudaErrorUnknown;
    queue.push_back({static_cast<char*>(dst), static_cast<const char*>(src), bytes, ++now});
    if (!is_pinned(kind == cudaMemcpyDeviceToHost ? dst : src)) run_until(now);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }

int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    static auto real = reinterpret_cast<decltype(&pthread_create)>(dlsym(RTLD_NEXT, "pthread_create"));
    ++threads;
    return fail_thread ? EAGAIN : real(t, a, f, x);
}
}

namespace fsb {
void fail(fs_status code, const std::string& msg) { throw FsError{code, msg}; }
void cuda_check(cudaError_t e, const char* what, const char*, int) {
    if (e != cudaSuccess) fail(FS_ERR_CUDA, what);
}
}  // namespace fsb

using namespace fsb;

size_t seed = 1;
// `n` bytes to the device and back through `S` (device arrays are host memory here).
void round_trip(HostStage& S, size_t n, const char* what) {
    std::vector<char> in(n), out(n), dev(n);
    for (size_t i = 0; i + 8 <= n; i += 8) std::memcpy(&in[i], &(seed += 0x9e3779b97f4a7c15u), 8);
    const size_t a = n / 3;
    S.to_device({{dev.data(), in.data(), a}, {dev.data() + a, in.data() + a, n - a}}, kStream);
    cudaStreamSynchronize(kStream);
    expect(dev == in, what);
    S.to_host({{out.data(), dev.data(), a}, {out.data() + a, dev.data() + a, n - a}}, kStream);
    expect(out == in, what);
}

constexpr size_t kMB = 1 << 20;

// Whatever calls of a copy fail, no staging memory is free or given back under it.
template <class F>
void failing(int& at, F copy) {
    for (int k : {0, 1, 2, 3, 5, 8, 13, 21, 34}) {
        at = -1;
        HostStage S;
        round_trip(S, 24 * kMB, "warm-up");
        copies = records = 0;
        at = k;
        try {
            copy(S);
        } catch (const FsError&) {
        }
        at = -1;
        round_trip(S, 24 * kMB, "after a failed copy");
    }
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    std::vector<char> host(24 * kMB), dev(24 * kMB);
    std::vector<HostCopy> out, in;
    for (size_t k = 0; k < 24; ++k) {
        out.push_back({host.data() + k * kMB, dev.data() + k * kMB, kMB - 8});
        in.push_back({dev.data() + k * kMB, host.data() + k * kMB, kMB - 8});
    }
    if (what == "failing copies") {
        failing(fail_copy, [&](HostStage& S) { S.to_host(out, kStream); });
        failing(fail_copy, [&](HostStage& S) { S.to_device(in, kStream); });
        failing(fail_record, [&](HostStage& S) { S.to_host(out, kStream); });
        failing(fail_record, [&](HostStage& S) { S.to_device(in, kStream); });
    } else if (what == "refused") {
        for (bool* b : {&fail_pin, &fail_event, &fail_thread}) {
            *b = true;
            {
                HostStage S;
                for (size_t n : {size_t(8), 40000 * size_t(8), 3 * kMB, 24 * kMB}) round_trip(S, n, "copy without what is refused");
            }
            *b = false;
            HostStage S;
            round_trip(S, 24 * kMB, "copy when it is granted again");
        }
        expect(pinned.empty(), "staging memory left over");
    } else if (what == "short lives") {
        for (int k = 0; k < 50; ++k) {  // one object after another
            HostStage S;
            round_trip(S, 2 * kMB, "copy of a short life");
        }
        expect(pins == 0 && threads == 0, "staging memory or threads for objects of one call");
        HostStage A;
        for (int k = 0; k < 30; ++k) {
            HostStage B;
            round_trip(B, 2 * kMB, "copy beside a long life");
        }
        expect(pins == 1, "no staging memory for many calls, or more than one piece");
        const int at = records;
        round_trip(A, 2 * kMB, "staged copy");
        expect(records > at, "a copy past its staging memory");
    } else {
        std::printf("no such scenario\n");
        return 2;
    }
    return bad ? 1 : 0;
}
