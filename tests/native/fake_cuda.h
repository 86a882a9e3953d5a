// A CUDA runtime without a GPU for tests of host code: device memory is host
// memory, copies happen at once, and every operation on a stream is recorded
// with the operations that stream order, events and host waits put before it
// and the bytes it touches, so that a test can ask which operations race.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <bitset>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

namespace fake {

constexpr int MAX_OPS = 4096;
typedef std::bitset<MAX_OPS> Ops;

struct Span {
    const char* lo;
    size_t n;
    bool write;
};
struct Op {
    std::string what;
    void* stream;
    std::thread::id thread;
    Ops before;
    std::vector<Span> spans;
    bool cooperative;
    bool overlap;      // may start before the operation ahead of it on the stream has ended
};

struct State {
    std::recursive_mutex mu;
    std::vector<Op> ops;
    std::map<void*, Ops> stream, event;    // what the next operation of a stream / a waiter of an event comes after
    Ops host;                              // what the host has waited for
    std::set<void*> live_streams, live_events;
    std::set<void*> busy, capturing;       // streams that report work, that are under capture
    std::map<char*, size_t> device;        // allocations
    std::vector<std::pair<const char*, size_t>> pinned;
    int mallocs = 0, current_device = 0;
    std::set<std::pair<const void*, int>> attributes;   // kernels whose shared memory limit was raised, by device
    std::map<std::string, int> calls;      // calls of each function
    std::string fail;                      // this function ...
    int fail_at = -1;                      // ... fails at this call (counted from 0; -1: never)
    int pause_us = 0;                      // length of a copy call and of a look-up of a driver function
    // pageable sources of copies that nobody has waited for, and what was in them:
    // where the device reads such memory itself, a copy may do so until then
    std::vector<std::pair<const char*, std::string>> unread;
    int gone = 0;                          // of them, those that were no longer the same when waited for
    // bytes that a kernel launch touches
    std::vector<Span> (*kernel_spans)(const void* kernel, void** args) = nullptr;
};
inline State& state() {
    static State s;
    return s;
}

// One call of function `name`: true when it is to fail.
inline bool fails(const char* name) {
    State& s = state();
    std::lock_guard<std::recursive_mutex> lock(s.mu);
    const int n = s.calls[name]++;
    return s.fail == name && s.fail_at == n;
}

inline void enqueue(const char* what, void* st, std::vector<Span> spans, bool cooperative = false,
                    bool overlap = false) {
    State& s = state();
    std::lock_guard<std::recursive_mutex> lock(s.mu);
    if (s.ops.size() >= MAX_OPS) abort();
    Op op{what, st, std::this_thread::get_id(), s.stream[st] | s.host, spans, cooperative, overlap};
    s.stream[st] = op.before;
    s.stream[st].set(s.ops.size());
    s.ops.push_back(op);
}

// Pairs of operations from number `from` on that touch the same bytes (of spans
// that `counts` picks), one of them writing, in no order.
inline int races(size_t from, bool (*counts)(const Span&) = nullptr) {
    State& s = state();
    int n = 0;
    for (size_t j = from; j < s.ops.size(); j++)
        for (size_t i = from; i < j; i++) {
            if (s.ops[j].before[i]) continue;
            bool hit = false;
            for (const Span& a : s.ops[i].spans)
                for (const Span& b : s.ops[j].spans)
                    if (!counts || (counts(a) && counts(b)))
                        hit = hit || ((a.write || b.write) && a.lo < b.lo + b.n && b.lo < a.lo + a.n);
            if (hit && n++ < 5) printf("race: %s (%zu) and %s (%zu)\n", s.ops[i].what.c_str(), i, s.ops[j].what.c_str(), j);
        }
    return n;
}

// The host waits for what was enqueued.
inline void waited() {
    for (auto& r : state().unread) state().gone += memcmp(r.first, r.second.data(), r.second.size()) != 0;
    state().unread.clear();
}

inline bool is_device(const void* p) {
    State& s = state();
    auto it = s.device.upper_bound((char*)p);
    if (it == s.device.begin()) return false;
    --it;
    return (char*)p < it->first + it->second;
}

inline void copy(const char* what, void* dst, const void* src, size_t n, void* st) {
    memcpy(dst, src, n);
    // a pageable source has been staged when the call returns
    std::vector<Span> v = {{(char*)dst, n, true}};
    State& s = state();
    bool pinned = is_device(src);
    for (auto& r : s.pinned) pinned = pinned || ((const char*)src >= r.first && (const char*)src < r.first + r.second);
    if (pinned) v.push_back({(const char*)src, n, false});
    else s.unread.push_back({(const char*)src, std::string((const char*)src, n)});
    enqueue(what, st, v);
}

}  // namespace fake
