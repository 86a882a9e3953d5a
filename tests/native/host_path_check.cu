// Host side of the collective API on a fake CUDA runtime: what it enqueues, in
// which order, what it allocates and what it leaves behind on errors.
// Usage: host_path_check SCENARIO
#include "fake_cuda.h"

#include <unistd.h>

#include <chrono>
#include <functional>

#include "spread.cuh"
using namespace gm;

static int bad = 0;
#define CHECK(x, ...)                                \
    do {                                             \
        if (!(x)) {                                  \
            if (bad++ < 10) {                        \
                printf("failed: %s: ", #x);          \
                printf(__VA_ARGS__);                 \
                printf("\n");                        \
            }                                        \
        }                                            \
    } while (0)

// Buffers of the calls of a test and what kernels other than tiles may touch.
struct Job_ {
    int P = 4;
    gpumpi_comm_t comm = nullptr;
    std::vector<std::vector<void*>> send, recv;
    std::vector<std::vector<char>> hsend, hrecv;   // pinned, rank by rank
    std::vector<void*> hs, hr;
    std::vector<gpumpi_coll_desc> descs;
    gpumpi_plan_t plan = nullptr;
};
static std::vector<fake::Span> g_buffers;   // device buffers of all jobs

typedef std::set<std::pair<const void*, const void*>> CallSet;
static std::vector<CallSet> g_launched;   // the calls of each launch, by their first rank's buffers

static std::vector<fake::Span> kernel_spans(const void* kernel, void** args) {
    if (kernel != (const void*)gpumpi_spread_kernel) return g_buffers;
    const SpreadArgs& a = *(const SpreadArgs*)args[0];
    g_launched.emplace_back();
    for (u32 i = 0; i < a.ncalls; i++) {
        const SpreadCall& c = a.ncalls == 1 ? a.one : a.calls[i];
        g_launched.back().insert({c.src[0], c.dst[0]});
    }
    std::vector<fake::Span> v;
    for (u32 i = 0; i < a.ncalls; i++) {
        if (a.ncalls > 1) v.push_back({(const char*)(a.calls + i), sizeof(SpreadCall), false});
        const SpreadCall& c = a.ncalls == 1 ? a.one : a.calls[i];
        v.push_back({(const char*)c.src, c.nsrc * sizeof(void*), false});
        v.push_back({(const char*)c.dst, c.ndst * sizeof(void*), false});
        for (u32 q = 0; q < c.nsrc; q++) v.push_back({c.src[q] + c.off, 16, false});
        for (u32 r = 0; r < c.ndst; r++) v.push_back({c.dst[r] + c.off, 16, true});
    }
    return v;
}

// A batched plan of `n` Allreduces of 4 ranks of `count` FP64 elements each, with pinned host buffers.
static Job_* make(int n, size_t count) {
    Job_* j = new Job_();
    CHECK(gpumpi_comm_create(j->P, &j->comm) == 0, "comm");
    j->send.resize(n);
    j->recv.resize(n);
    for (int i = 0; i < n; i++)
        for (int r = 0; r < 2 * j->P; r++) {
            void* d = nullptr;
            cudaMalloc(&d, count * 8);
            g_buffers.push_back({(char*)d, count * 8, true});
            (r < j->P ? j->send : j->recv)[i].push_back(d);
            std::vector<char> h(count * 8, (char)(r + i));
            (r < j->P ? j->hsend : j->hrecv).push_back(h);
        }
    for (auto* side : {&j->hsend, &j->hrecv})
        for (auto& h : *side) {
            fake::state().pinned.push_back({h.data(), h.size()});
            (side == &j->hsend ? j->hs : j->hr).push_back(h.data());
        }
    for (int i = 0; i < n; i++) {
        gpumpi_coll_desc d;
        memset(&d, 0, sizeof(d));
        d.comm = j->comm;
        d.op = GPUMPI_COLL_ALLREDUCE;
        d.dtype = MPI_DOUBLE;
        d.redop = GPUMPI_OP_SUM;
        d.count = count;
        d.sendbufs = j->send[i].data();
        d.recvbufs = j->recv[i].data();
        j->descs.push_back(d);
    }
    CHECK(gpumpi_plan_create(j->descs.data(), n, 64, 1, &j->plan) == 0, "plan: %s", gpumpi_last_error());
    return j;
}
static int run_host(Job_* j, cudaStream_t st) {
    return gpumpi_plan_run_host(j->plan, j->hs.data(), j->hr.data(), st, nullptr, nullptr);
}
static cudaStream_t stream() {
    cudaStream_t st = nullptr;
    cudaStreamCreateWithFlags(&st, 0);
    return st;
}
static int streams_used(size_t from) {
    std::set<void*> used;
    for (size_t i = from; i < fake::state().ops.size(); i++) used.insert(fake::state().ops[i].stream);
    return (int)used.size();
}

static const size_t LARGE = 1 << 16, SMALL = 1 << 10;   // elements: 4 MiB and more in 2 calls, less

// A host-buffer call allocates no device memory, and its tile lists have arrived before a launch reads them.
static void tables() {
    Job_* j = make(3, LARGE);
    const size_t from = fake::state().ops.size();
    const int mallocs = fake::state().mallocs;
    CHECK(run_host(j, stream()) == 0, "%s", gpumpi_last_error());
    CHECK(fake::state().mallocs == mallocs, "%d allocations", fake::state().mallocs - mallocs);
    CHECK(streams_used(from) == 3, "%d streams", streams_used(from));
    CHECK(fake::races(from) == 0, "races");
}

// The tile lists have arrived before a launch reads them, also where the first
// call does not use them (results over its inputs) and the next one is on
// another stream.
static bool in_tables(const fake::Span& a) {
    for (const fake::Span& b : g_buffers)
        if (a.lo >= b.lo && a.lo < b.lo + b.n) return false;
    return fake::is_device(a.lo);
}
static void uploaded() {
    Job_* j = make(3, LARGE);
    const size_t from = fake::state().ops.size();
    CHECK(gpumpi_plan_run_host(j->plan, j->hs.data(), j->hs.data(), stream(), nullptr, nullptr) == 0, "first");
    CHECK(run_host(j, stream()) == 0, "%s", gpumpi_last_error());
    CHECK(streams_used(from) == 4 && fake::races(from, in_tables) == 0, "%d streams", streams_used(from));
}

// Where the streams of the groups cannot be had, one after another; the next call tries again.
static void retry() {
    Job_* j = make(3, LARGE);
    cudaStream_t st = stream();
    fake::state().fail = "cudaStreamCreateWithFlags";
    fake::state().fail_at = fake::state().calls["cudaStreamCreateWithFlags"] + 1;
    const size_t streams = fake::state().live_streams.size(), events = fake::state().live_events.size();
    size_t from = fake::state().ops.size();
    CHECK(run_host(j, st) == 0, "%s", gpumpi_last_error());
    CHECK(streams_used(from) == 1 && fake::races(from) == 0, "%d streams", streams_used(from));
    CHECK(fake::state().live_streams.size() == streams && fake::state().live_events.size() <= events + 1, "left behind");
    from = fake::state().ops.size();
    CHECK(run_host(j, st) == 0, "%s", gpumpi_last_error());
    CHECK(streams_used(from) == 3 && fake::races(from) == 0, "%d streams", streams_used(from));
}

// Calls of one plan on different streams: each ends before the next one starts.
static void order() {
    for (size_t count : {LARGE, SMALL}) {
        Job_* j = make(3, count);
        const size_t from = fake::state().ops.size();
        for (int i = 0; i < 3; i++) CHECK(run_host(j, stream()) == 0, "%s", gpumpi_last_error());
        CHECK(fake::races(from) == 0, "races of %zu elements", count);
    }
}

// Calls of one plan from two threads on one stream do not mix, whatever their form.
static void turns() {
    for (size_t count : {LARGE, SMALL}) {
        Job_* j = make(3, count);
        cudaStream_t st = stream();
        const size_t from = fake::state().ops.size();
        fake::state().pause_us = 200;
        std::vector<std::thread> threads;
        for (int t = 0; t < 2; t++)
            threads.emplace_back([&] {
                for (int i = 0; i < 3; i++) CHECK(run_host(j, st) == 0, "%s", gpumpi_last_error());
            });
        for (auto& t : threads) t.join();
        fake::state().pause_us = 0;
        // a call's operations: the same number each, by one thread
        const std::vector<fake::Op>& ops = fake::state().ops;
        const size_t each = (ops.size() - from - (count == LARGE)) / 6;   // and the tile lists, with the first
        for (size_t i = 0; i < 6; i++)
            for (size_t k = 0; k < each; k++) {
                const size_t at = from + (count == LARGE) + i * each;
                CHECK(ops[at + k].thread == ops[at].thread, "call %zu of %zu elements", i, count);
            }
        CHECK(fake::races(from) == 0, "races of %zu elements", count);
    }
}

// The first calls of a process, of two plans from two threads: both go in groups.
static void first_calls() {
    Job_* jobs[2] = {make(3, LARGE), make(3, LARGE)};
    cudaStream_t streams[2] = {stream(), stream()};
    const size_t from = fake::state().ops.size();
    fake::state().pause_us = 2000;
    std::vector<std::thread> threads;
    for (int t = 0; t < 2; t++)
        threads.emplace_back([&, t] {
            std::this_thread::sleep_for(std::chrono::microseconds(1000 * t));
            CHECK(run_host(jobs[t], streams[t]) == 0, "%s", gpumpi_last_error());
        });
    for (auto& t : threads) t.join();
    fake::state().pause_us = 0;
    CHECK(streams_used(from) == 6, "%d streams", streams_used(from));
}

// A captured plan of one launch replays its graph on an idle stream and is
// launched behind other work or under capture; one of several launches is a graph always.
static void captured() {
    Job_* j = make(3, SMALL);
    cudaStream_t st = stream();
    auto launched = [&](gpumpi_plan_t p) {
        const size_t from = fake::state().ops.size();
        const uint64_t count = gpumpi_kernel_launches();
        CHECK(gpumpi_plan_launch(p, st) == 0, "%s", gpumpi_last_error());
        CHECK(gpumpi_kernel_launches() > count, "launches");
        return fake::state().ops.size() == from + 1 ? fake::state().ops[from].what : std::string("?");
    };
    CHECK(launched(j->plan) == "launch", "before the capture");
    const uint64_t count = gpumpi_kernel_launches();
    CHECK(gpumpi_plan_capture(j->plan, nullptr) == 0 && gpumpi_kernel_launches() == count, "%s", gpumpi_last_error());
    CHECK(launched(j->plan) == "graph", "idle");
    fake::state().busy.insert(st);
    CHECK(launched(j->plan) == "launch", "busy");
    fake::state().busy.clear();
    fake::state().capturing.insert(st);
    CHECK(launched(j->plan) == "launch", "under capture");
    fake::state().capturing.clear();
    CHECK(launched(j->plan) == "graph", "idle again");
    CHECK(gpumpi_plan_set_sync(j->plan, 1) == 0 && gpumpi_plan_set_sync(j->plan, 0) == 0, "set_sync");
    CHECK(launched(j->plan) == "launch", "the graph has been dropped");
    j->descs[1].sendbufs = j->descs[0].recvbufs;   // a second level
    gpumpi_plan_t p = nullptr;
    CHECK(gpumpi_plan_create(j->descs.data(), 3, 64, 1, &p) == 0 && gpumpi_plan_capture(p, nullptr) == 0, "%s",
          gpumpi_last_error());
    CHECK(launched(p) == "graph", "levels, idle");
    fake::state().busy.insert(st);
    CHECK(launched(p) == "graph", "levels, busy");
    gpumpi_plan_destroy(p);
}

// The tuner measures again what a file has from before some schedules ran as
// tiles, and reads what it wrote itself.
static void tuner_file() {
    Job_* j = make(1, SMALL);
    char path[] = "/tmp/host_path_tuneXXXXXX";
    FILE* f = fdopen(mkstemp(path), "w");
    for (int t : {64, 128, 256, 512, 1024}) fprintf(f, "fake GPU|3 13 2 4 %zu %d|2 0.01\n", SMALL, t);
    fclose(f);
    gpumpi_tune_opts opts = {1, path, 0};
    const uint64_t before = gpumpi_kernel_launches();
    int threads = 0, algo = 0;
    CHECK(gpumpi_autotune(j->descs.data(), 1, &opts, nullptr, &threads, &algo) == 0, "%s", gpumpi_last_error());
    CHECK(algo == 1 && gpumpi_kernel_launches() > before, "schedule %d", algo);   // all take as long: the first
    const uint64_t once = gpumpi_kernel_launches();
    CHECK(gpumpi_autotune(j->descs.data(), 1, &opts, nullptr, &threads, &algo) == 0, "%s", gpumpi_last_error());
    CHECK(algo == 1 && gpumpi_kernel_launches() == once, "schedule %d", algo);
    remove(path);
}

// A call without a plan waits once, for its results; its tables arrive in the
// stream's order, ahead of its first launch, which does not overlap them.
static void one_shot_calls() {
    Job_* j = make(3, SMALL);
    for (int dependent : {0, 1}) {
        if (dependent) j->descs[1].sendbufs = j->descs[0].recvbufs;
        for (auto call : {gpumpi_coll_plain, gpumpi_coll_batched}) {
            cudaStream_t st = stream();
            const size_t from = fake::state().ops.size();
            const int waits = fake::state().calls["cudaStreamSynchronize"];
            CHECK(call(j->descs.data(), 3, 64, st) == 0, "%s", gpumpi_last_error());
            CHECK(fake::state().calls["cudaStreamSynchronize"] == waits + 1, "%d waits",
                  fake::state().calls["cudaStreamSynchronize"] - waits);
            bool first = true;
            for (size_t i = from; i < fake::state().ops.size(); i++) {
                const fake::Op& op = fake::state().ops[i];
                if (op.what != "launch") continue;
                CHECK(op.stream == st && op.before[from] && op.overlap == !first, "launch %zu", i - from);
                first = false;
            }
            CHECK(!first && fake::races(from) == 0, "dependent %d", dependent);
        }
    }
}

// What copies to the device read from pageable memory stays as it is until the
// stream has been waited for.
static void images() {
    Job_* j = make(3, LARGE);
    cudaStream_t st = stream();
    fake::state().unread.clear();   // the communicator's and the plan's, waited for by what came after
    fake::state().gone = 0;
    CHECK(run_host(j, st) == 0, "%s", gpumpi_last_error());
    CHECK(fake::state().unread.size() == 1, "%zu pageable copies", fake::state().unread.size());   // the tile lists
    cudaStreamSynchronize(st);
    CHECK(fake::state().gone == 0, "a group's tile lists");
    fake::state().gone = 0;
    CHECK(gpumpi_coll_batched(j->descs.data(), 3, 64, st) == 0, "%s", gpumpi_last_error());
    CHECK(fake::state().gone == 0 && fake::state().unread.empty(), "a call's tables");
}

// A call that fails half way reports it, and nothing that it put on other streams outlives a wait for the caller's.
static void errors() {
    int failed = 0;
    for (const char* what : {"cudaMemcpyAsync", "cudaLaunchKernelExC", "cudaEventRecord", "cudaStreamWaitEvent"}) {
        Job_* j = make(3, LARGE);
        cudaStream_t st = stream();
        CHECK(run_host(j, st) == 0, "%s", gpumpi_last_error());
        const int first = fake::state().calls[what];
        CHECK(run_host(j, st) == 0, "%s", gpumpi_last_error());
        const int n = fake::state().calls[what] - first;
        for (int k = 0; k < n; k++) {
            const size_t from = fake::state().ops.size();
            fake::state().fail = what;
            fake::state().fail_at = fake::state().calls[what] + k;
            const int rc = run_host(j, st);
            fake::state().fail_at = -1;
            failed += rc != 0;
            CHECK(rc == GPUMPI_ECUDA, "%s call %d: %d", what, k, rc);
            const fake::Ops done = fake::state().stream[st] | fake::state().host;
            for (size_t i = from; i < fake::state().ops.size(); i++) CHECK(done[i], "%s call %d: operation %zu", what, k, i);
            CHECK(run_host(j, st) == 0 && fake::races(from) == 0, "%s call %d: the next call", what, k);
        }
    }
    CHECK(failed > 30, "%d", failed);
}

// A plan of calls that use each other's results: a launch for each level, none of which needs all its blocks
// on the GPU at once.
static void levels() {
    Job_* j = make(1, SMALL);
    std::vector<gpumpi_coll_desc> d(5, j->descs[0]);
    for (int i = 1; i < 5; i += 2) std::swap(d[i].sendbufs, d[i].recvbufs);
    gpumpi_plan_t p = nullptr;
    CHECK(gpumpi_plan_create(d.data(), 5, 64, 1, &p) == 0, "%s", gpumpi_last_error());
    cudaStream_t st = stream();
    const size_t from = fake::state().ops.size();
    const uint64_t counted = gpumpi_kernel_launches();
    CHECK(gpumpi_plan_launch(p, st) == 0, "%s", gpumpi_last_error());
    CHECK(fake::state().ops.size() - from == 5 && gpumpi_kernel_launches() - counted == 5, "%zu launches",
          fake::state().ops.size() - from);
    for (size_t i = from; i < fake::state().ops.size(); i++)
        CHECK(!fake::state().ops[i].cooperative && fake::state().ops[i].stream == st, "launch %zu", i - from);
}

// The levels of random lists of Allreduces over one piece of memory: as few as their conflicts allow.
static void random_levels() {
    unsigned long long x = 12345;
    auto rnd = [&](int n) { return (int)((x = x * 6364136223846793005ull + 1442695040888963407ull) >> 33) % n; };
    void* mem = nullptr;
    cudaMalloc(&mem, 1 << 16);
    gpumpi_comm_t comm = nullptr;
    CHECK(gpumpi_comm_create(2, &comm) == 0, "comm");
    for (int it = 0; it < 300; it++) {
        const int n = 1 + rnd(12), room = 8 << rnd(9);
        std::vector<std::vector<void*>> at(2 * n);
        std::vector<gpumpi_coll_desc> d(n);
        for (int i = 0; i < n; i++) {
            memset(&d[i], 0, sizeof(d[i]));
            d[i].comm = comm;
            d[i].op = GPUMPI_COLL_ALLREDUCE;
            d[i].dtype = MPI_DOUBLE;
            d[i].redop = GPUMPI_OP_SUM;
            d[i].count = 1 + rnd(1 + room / 8);
            for (int k = 0; k < 4; k++) at[2 * i + k / 2].push_back((char*)mem + 8 * rnd(room));
            d[i].sendbufs = at[2 * i].data();
            d[i].recvbufs = at[2 * i + 1].data();
        }
        auto conflict = [&](int i, int j) {
            for (int a = 0; a < 4; a++)
                for (int b = 0; b < 4; b++) {
                    const char *p = (char*)at[2 * i + a / 2][a % 2], *q = (char*)at[2 * j + b / 2][b % 2];
                    if ((a >= 2 || b >= 2) && p < q + 8 * d[j].count && q < p + 8 * d[i].count) return true;
                }
            return false;
        };
        std::vector<int> level(n, 0);
        std::vector<CallSet> want;
        for (int i = 0; i < n; i++) {
            for (int j = 0; j < i; j++)
                if (conflict(i, j)) level[i] = std::max(level[i], level[j] + 1);
            if ((int)want.size() <= level[i]) want.resize(level[i] + 1);
            want[level[i]].insert({at[2 * i][0], at[2 * i + 1][0]});
        }
        gpumpi_plan_t p = nullptr;
        CHECK(gpumpi_plan_create(d.data(), n, 64, 1, &p) == 0, "%s", gpumpi_last_error());
        g_launched.clear();
        CHECK(gpumpi_plan_launch(p, nullptr) == 0, "%s", gpumpi_last_error());
        CHECK(g_launched == want, "list %d: %zu levels, %zu expected", it, g_launched.size(), want.size());
        gpumpi_plan_destroy(p);
    }
}

// Creating a long plan of dependent calls takes no more than a few times as long as one of independent calls.
static void long_plans() {
    const int P = 256, n = 2000;
    void* mem = nullptr;
    cudaMalloc(&mem, (size_t)P * (n + 1) * 8);
    gpumpi_comm_t comm = nullptr;
    CHECK(gpumpi_comm_create(P, &comm) == 0, "comm");
    double took[2];
    for (int dependent = 0; dependent < 2; dependent++) {
        std::vector<std::vector<void*>> at(n + 1);
        for (int i = 0; i <= n; i++)
            for (int r = 0; r < P; r++) at[i].push_back((char*)mem + ((size_t)(dependent ? i % 2 : i) * P + r) * 8);
        std::vector<gpumpi_coll_desc> d(n);
        for (int i = 0; i < n; i++) {
            memset(&d[i], 0, sizeof(d[i]));
            d[i].comm = comm;
            d[i].op = GPUMPI_COLL_ALLREDUCE;
            d[i].dtype = MPI_DOUBLE;
            d[i].redop = GPUMPI_OP_SUM;
            d[i].count = 1;
            d[i].sendbufs = dependent ? at[i].data() : nullptr;
            d[i].recvbufs = at[i + 1].data();
        }
        gpumpi_plan_t p = nullptr;
        const auto t0 = std::chrono::steady_clock::now();
        CHECK(gpumpi_plan_create(d.data(), n, 64, 1, &p) == 0, "%s", gpumpi_last_error());
        took[dependent] = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        CHECK(gpumpi_plan_launch_ordered(p) == !dependent, "form");
        gpumpi_plan_destroy(p);
    }
    printf("independent %.3f s, dependent %.3f s\n", took[0], took[1]);
    CHECK(took[1] < 10 * took[0] + 0.2, "%.3f s, %.3f s", took[0], took[1]);
}

// A plan made on a second device raises the kernels' shared memory limit there too.
static void devices() {
    for (int dev : {0, 1, 0, 2}) {
        fake::state().current_device = dev;
        make(1, SMALL);
        CHECK(fake::state().attributes.count({(const void*)gpumpi_spread_kernel, dev}) == 1, "device %d", dev);
    }
}

// A plan that cannot be made leaves no device memory behind.
static void failed_plans() {
    Job_* j = make(3, SMALL);
    for (const char* what : {"cudaMalloc", "cudaMemcpy", "cudaStreamSynchronize", "cudaGetDevice",
                             "cudaOccupancyMaxActiveBlocksPerMultiprocessor"})
        for (int batched : {0, 1}) {
            const size_t before = fake::state().device.size();
            gpumpi_plan_t p = nullptr;
            int first = fake::state().calls[what];
            CHECK(gpumpi_plan_create(j->descs.data(), 3, 64, batched, &p) == 0, "%s", gpumpi_last_error());
            gpumpi_plan_destroy(p);
            const int n = fake::state().calls[what] - first;
            CHECK(n > 0, "%s is not called", what);
            fake::state().fail = what;
            for (int k = 0; k < n; k++) {
                fake::state().fail_at = fake::state().calls[what] + k;
                p = nullptr;
                const int rc = gpumpi_plan_create(j->descs.data(), 3, 64, batched, &p);
                fake::state().fail_at = -1;
                CHECK(rc == 0 || p == nullptr, "%s call %d", what, k);
                if (rc == 0) gpumpi_plan_destroy(p);   // the rank blocks' staging is sized without it
                CHECK(fake::state().device.size() == before, "%s call %d: memory left", what, k);
            }
        }
}

int main(int argc, char** argv) {
    const std::map<std::string, std::function<void()>> scenarios = {
        {"tables", tables}, {"uploaded", uploaded}, {"retry", retry}, {"order", order}, {"turns", turns},
        {"first_calls", first_calls}, {"captured", captured}, {"tuner_file", tuner_file},
        {"one_shot_calls", one_shot_calls}, {"images", images}, {"errors", errors},
        {"levels", levels}, {"random_levels", random_levels}, {"long_plans", long_plans},
        {"devices", devices}, {"failed_plans", failed_plans}};
    fake::state().kernel_spans = kernel_spans;
    scenarios.at(argc > 1 ? argv[1] : "")();
    printf("%s bad %d\n", argv[1], bad);
    return bad != 0;
}
