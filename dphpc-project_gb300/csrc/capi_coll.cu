// Host-driven collectives: communicators and plans that run a list of
// collective calls with one kernel launch per call ("plain") or with as few as
// their dependences allow ("batched").  Calls that need no flag rounds run as
// independent tiles over the whole GPU (spread.cuh); the others as thread
// blocks, one for each rank, which run the device schedules of the MPI_* calls
// of converted programs (coll.cu), a batched list in one cooperative launch.
// Results are the same bits in every form.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <memory>
#include <mutex>
#include <vector>

#include "gpumpi.h"
#include "hostjob.h"
#include "rt.cuh"
#include "spread.cuh"

extern __device__ MPI_Op_impl gm_builtin_ops[GPUMPI_NUM_BUILTIN_OPS];

namespace gm {

struct DevDesc {
    int op;
    int dtype;
    int redop;
    int root;
    u64 count;
    int comm;       // index into the plan's communicator table
    int esize;
    int algo;
    int sync;       // 1: flag rounds even when the launch is launch-ordered
    void** sbufs;   // [P] device array
    void** rbufs;   // [P]
    const Pub* pub; // [P] buffer table of the launch-ordered forms (nullptr: none)
};

struct DevComm {
    MPI_Comm_impl* handles;   // [P] per-rank handles (sequence numbers persist)
    int size;
    int pad;
};

struct PlanArgs {
    Job* job;
    const DevDesc* descs;
    const int* comm_first;    // [ncomm + 1]: descriptor range of each communicator
    const int* slot_comm;     // [nslots], nullptr = every block in communicator 0
    const int* slot_rank;     // [nslots], nullptr = rank is blockIdx.x
    const DevComm* comms;
    int ordered;              // 1: the launch-ordered forms (calls touch disjoint memory)
    int pad;
};

static __device__ int run_desc(const DevDesc& d, MPI_Comm_impl* comm, int P, int rank, int ordered, int tid,
                               int T) {
    CollArgs a;
    memset(&a, 0, sizeof(a));
    a.comm = comm;
    a.root = d.root;
    a.algo = d.algo;
    a.ssize = a.rsize = d.esize;
    a.dtype = (MPI_Datatype)d.dtype;
    a.op = &gm_builtin_ops[d.redop];
    a.opi = d.redop;
    a.ufn = nullptr;
    const void* sb = d.sbufs ? ldcg(&d.sbufs[rank]) : nullptr;
    void* rb = d.rbufs ? ldcg(&d.rbufs[rank]) : nullptr;
    if (ordered && d.pub && !d.sync) {
        a.sbuf = sb;
        a.rbuf = rb;
        switch (d.op) {
            case GPUMPI_COLL_BCAST:
                if (d.algo == 2) break;   // the tree forwards copies made in this launch: flag rounds
                a.count = d.count * d.esize;
                return coll_lo_bcast(a, d.pub, P, rank, tid, T);
            case GPUMPI_COLL_REDUCE:
                a.count = d.count;
                return coll_lo_reduce(a, d.pub, P, rank, tid, T);
            case GPUMPI_COLL_ALLREDUCE:
                a.count = d.count;
                return coll_lo_allreduce(a, d.pub, P, rank, tid, T);
            case GPUMPI_COLL_ALLTOALL:
            case GPUMPI_COLL_ALLGATHER:
                a.count = d.count;
                return coll_lo_alltoall(a, d.pub, P, rank, d.op == GPUMPI_COLL_ALLGATHER, tid, T);
            default: break;   // a barrier keeps its flag round
        }
    }
    switch (d.op) {
        case GPUMPI_COLL_BARRIER: return coll_barrier(comm, tid, T);
        case GPUMPI_COLL_BCAST:
            a.rbuf = rb;
            a.count = d.count * d.esize;
            return coll_bcast(a, tid, T);
        case GPUMPI_COLL_REDUCE:
            a.sbuf = sb;
            a.rbuf = rb;
            a.count = d.count;
            return coll_reduce(a, tid, T);
        case GPUMPI_COLL_ALLREDUCE:
            a.sbuf = sb;
            a.rbuf = rb;
            a.count = d.count;
            return coll_allreduce(a, tid, T);
        case GPUMPI_COLL_ALLTOALL:
            a.sbuf = sb;
            a.rbuf = rb;
            a.a0 = (long long)d.count;
            a.a1 = (long long)d.count;
            return coll_alltoallv(a, tid, T);
        case GPUMPI_COLL_ALLGATHER:
            a.sbuf = sb;
            a.rbuf = rb;
            a.a0 = (long long)d.count;
            a.a1 = (long long)d.count;
            return coll_allgatherv(a, tid, T);
        default: return MPI_ERR_ARG;
    }
}

extern "C" __global__ void __launch_bounds__(1024) gpumpi_plan_kernel(PlanArgs A) {
    BlockCtx& b = bctx();
    const int slot = blockIdx.x;
    const int c = A.slot_comm ? A.slot_comm[slot] : 0;
    const int rank = A.slot_rank ? A.slot_rank[slot] : slot;
    if (threadIdx.x == 0) {
        b.job = A.job;
        b.priv = nullptr;
        b.rank = rank;
        b.slot = slot;
        b.T = (int)blockDim.x;
        b.leader_mode = 0;
        b.in_call = 0;
        b.bulk_broken = 0;
        b.lazy_n = 0;
        b.sc_handle = nullptr;
        b.mb_cluster = 0;
        b.mb_local = nullptr;
        b.cl_n = 1;
        b.cl_rank = 0;
    }
    __syncthreads();
    MPI_Comm_impl* comm = &A.comms[c].handles[rank];
    const int tid = (int)threadIdx.x, T = (int)blockDim.x;
    const int P = A.comms[c].size;
    for (int i = A.comm_first[c]; i < A.comm_first[c + 1]; i++) {
        if (run_desc(A.descs[i], comm, P, rank, A.ordered, tid, T) != MPI_SUCCESS) break;
    }
}

}  // namespace gm

using namespace gm;

// ------------------------------------------------------------------ host side
struct gpumpi_comm_s {
    int n;
    char* base;          // device allocation
    DevComm* dcomm;      // device DevComm
    DevComm hcomm;
};

// The calls of a plan in groups, for host-buffer calls that copy in, run and
// copy out one group after another on three streams.
struct HostPipe {
    enum State { NEW, READY, NONE } state = NEW;   // NONE: no two groups, or calls that share device memory
    std::vector<std::vector<int>> groups;  // calls (creation order) of each group
    std::vector<SpreadArgs> tiles;
    std::vector<char> image;               // of the tile lists, which a copy from it may still read
    cudaStream_t in = nullptr, out = nullptr;
    cudaEvent_t begin = nullptr, end = nullptr;
    std::vector<cudaEvent_t> arrived, ran;
    void drop() {
        for (auto e : arrived) cudaEventDestroy(e);
        for (auto e : ran) cudaEventDestroy(e);
        if (begin) cudaEventDestroy(begin);
        if (end) cudaEventDestroy(end);
        if (in) cudaStreamDestroy(in);
        if (out) cudaStreamDestroy(out);
        arrived.clear();
        ran.clear();
        groups.clear();
        tiles.clear();
        image.clear();
        begin = end = nullptr;
        in = out = nullptr;
    }
    ~HostPipe() { drop(); }
};

struct gpumpi_plan_s {
    int ndesc;
    int ncomm;
    int batched;
    int threads;
    size_t smem;
    char* base = nullptr;             // device allocation
    std::vector<char> image;          // what a stream's copy to it may still read
    PlanArgs batch_args;              // batched launch
    std::vector<PlanArgs> plain_args; // one per descriptor
    std::vector<int> plain_grid;
    std::vector<int> plain_threads;   // threads per rank of each plain launch
    std::vector<size_t> plain_smem;   // dynamic shared memory of each plain launch
    int total_slots;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<gpumpi_coll_desc> descs;   // host copies for the host-buffer path
    std::vector<std::vector<void*>> sb, rb;
    int independent = 0;                   // calls touch disjoint memory and include no barrier
    int sync_mode = 0;                     // 0 automatic, 1 flag rounds for every call
    std::vector<int> plain_op;             // collective of each plain launch
    // spread form (spread.cuh) of a batched launch, one launch for each level of
    // its calls, and of the launch-ordered plain launches that it covers
    bool batch_spread = false;
    std::vector<SpreadArgs> batch_tiles;
    std::vector<char> plain_spread;
    std::vector<SpreadArgs> plain_tiles;
    std::mutex pipe_mu;                    // host-buffer calls of one plan enqueue one after another
    HostPipe pipe;                         // filled in by the first one
    char* pipe_base = nullptr;             // part of `base` for the groups' tile lists
    size_t pipe_bytes = 0;
    cudaEvent_t host_done = nullptr;       // end of the last host-buffer call, the next one starts after it
    ~gpumpi_plan_s() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (host_done) cudaEventDestroy(host_done);
        if (base) cudaFree(base);
    }
};

namespace {

std::atomic<unsigned long long> g_launches{0};

struct ApiJob {
    Job* djob = nullptr;
    int* status = nullptr;
    char* err = nullptr;
};
ApiJob g_api;

#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            char m_[300];                                                                 \
            snprintf(m_, sizeof(m_), "%s: %s", #call, cudaGetErrorString(e_));            \
            set_last_error(m_);                                                           \
            return GPUMPI_ECUDA;                                                          \
        }                                                                                 \
    } while (0)

int spread_attributes();

int api_job() {
    int rc = spread_attributes();
    if (rc) return rc;
    if (g_api.djob) return GPUMPI_OK;
    // the plan kernel streams through L2 (ld.global.cg) and stages bulk copies
    // in shared memory: prefer the largest shared-memory carve-out
    CK(cudaFuncSetAttribute((const void*)gpumpi_plan_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                            (int)cudaSharedmemCarveoutMaxShared));
    Job hj;
    memset(&hj, 0, sizeof(hj));
    char* mem = nullptr;
    CK(cudaMalloc(&mem, sizeof(Job) + 64 + 256));
    CK(cudaMemset(mem, 0, sizeof(Job) + 64 + 256));
    hj.id = -1;
    hj.timeout_ns = 30ull * 1000000000ull;
    hj.status = (int*)(mem + sizeof(Job));
    hj.err_msg = mem + sizeof(Job) + 64;
    CK(cudaMemcpy(mem, &hj, sizeof(Job), cudaMemcpyHostToDevice));
    g_api.djob = (Job*)mem;
    g_api.status = hj.status;
    g_api.err = hj.err_msg;
    return GPUMPI_OK;
}

int esize_of(int dtype) {
    switch (dtype) {
        case MPI_CHAR: case MPI_SIGNED_CHAR: case MPI_UNSIGNED_CHAR: case MPI_BYTE: case MPI_INT8_T:
        case MPI_UINT8_T: case MPI_C_BOOL: return 1;
        case MPI_SHORT: case MPI_UNSIGNED_SHORT: case MPI_INT16_T: case MPI_UINT16_T: return 2;
        case MPI_INT: case MPI_UNSIGNED: case MPI_FLOAT: case MPI_INT32_T: case MPI_UINT32_T: return 4;
        case MPI_LONG: case MPI_LONG_LONG_INT: case MPI_LONG_LONG: case MPI_UNSIGNED_LONG:
        case MPI_UNSIGNED_LONG_LONG: case MPI_DOUBLE: case MPI_INT64_T: case MPI_UINT64_T: return 8;
        default: return -1;
    }
}

// Bytes a rank sends / receives for a descriptor.
void desc_bytes(const gpumpi_coll_desc& d, int P, size_t* in, size_t* out) {
    size_t e = (size_t)esize_of(d.dtype) * d.count;
    switch (d.op) {
        case GPUMPI_COLL_BCAST: *in = e; *out = e; break;
        case GPUMPI_COLL_REDUCE:
        case GPUMPI_COLL_ALLREDUCE: *in = e; *out = e; break;
        case GPUMPI_COLL_ALLTOALL: *in = e * P; *out = e * P; break;
        case GPUMPI_COLL_ALLGATHER: *in = e; *out = e * P; break;
        default: *in = *out = 0;
    }
}

// Bytes a host-buffer call copies for a descriptor of P ranks, both ways.
size_t host_bytes(const gpumpi_coll_desc& d, int P, size_t* in, size_t* out) {
    desc_bytes(d, P, in, out);
    if (d.op != GPUMPI_COLL_BCAST) *in *= P;
    if (d.op != GPUMPI_COLL_REDUCE) *out *= P;
    return *in + *out;
}

constexpr int PIPE_GROUPS = 8;
constexpr size_t PIPE_MIN_BYTES = 4u << 20;   // below, the groups' launches and events cost more than the overlap gives

// Levels of the calls of a list: a call is one level above the highest earlier
// call that it shares memory with, one of the two writing it, so the calls of
// one level touch disjoint memory.  Each call's spans: the bytes each rank
// reads and writes (Bcast: the root's buffer is read, the others written).
// Spans of one call never conflict with each other here (in-place forms are
// the schedules' concern).  Spans are sorted by start and compared with the
// spans still open, up to the first conflict: lists without one are done.  In
// the others the spans' ends cut memory into pieces, and each call in turn
// comes after the last writer of every piece it uses and after the readers
// since then of every piece it writes.  That takes time in proportion to the
// spans, where all pairs of conflicting calls take its square (creating a plan
// of 2000 Allreduces of 256 ranks that ping-pong between two buffers: 7.2 s by
// pairs, 0.18 s so, 0.11 s when they are independent).  Returns the number of levels, or 0
// when the list holds a barrier or is too long to be levelled.  One level means
// that the plan kernel may run every call in its launch-ordered form.
// fill_inputs: what a call reads counts as written (a host-buffer call copies
// it in).
constexpr int MAX_LEVEL_CALLS = 2048;
constexpr size_t MAX_LEVEL_PIECES = 1u << 26;   // pieces of all spans, 0.2 s
int plan_levels(const gpumpi_coll_desc* descs, int ndesc, std::vector<int>& level, bool fill_inputs = false) {
    struct Span {
        uintptr_t lo, hi;
        int call, w;
    };
    std::vector<Span> v;
    for (int i = 0; i < ndesc; i++) {
        const gpumpi_coll_desc& d = descs[i];
        if (d.op == GPUMPI_COLL_BARRIER) return 0;
        const int P = d.comm->n;
        const size_t e = (size_t)esize_of(d.dtype) * d.count;
        auto add = [&](void* const* tab, int r, size_t bytes, int w) {
            const void* p = tab ? tab[r] : nullptr;
            if (p && bytes) v.push_back({(uintptr_t)p, (uintptr_t)p + bytes, i, w || fill_inputs});
        };
        for (int r = 0; r < P; r++) {
            switch (d.op) {
                case GPUMPI_COLL_BCAST: add(d.recvbufs, r, e, r != d.root); break;
                case GPUMPI_COLL_REDUCE:
                    add(d.sendbufs ? d.sendbufs : d.recvbufs, r, e, 0);
                    if (r == d.root) add(d.recvbufs, r, e, 1);
                    break;
                case GPUMPI_COLL_ALLREDUCE:
                    add(d.sendbufs, r, e, 0);
                    add(d.recvbufs, r, e, 1);
                    break;
                case GPUMPI_COLL_ALLTOALL:
                    add(d.sendbufs, r, e * P, 0);
                    add(d.recvbufs, r, e * P, 1);
                    break;
                case GPUMPI_COLL_ALLGATHER:
                    add(d.sendbufs, r, e, 0);
                    add(d.recvbufs, r, e * P, 1);
                    break;
                default: break;
            }
        }
    }
    std::sort(v.begin(), v.end(), [](const Span& a, const Span& b) { return a.lo < b.lo; });
    level.assign(ndesc, 0);
    bool conflict = false;
    std::vector<Span> open;
    for (size_t i = 0; i < v.size() && !conflict; i++) {
        const Span& x = v[i];
        size_t k = 0;
        for (size_t j = 0; j < open.size(); j++)
            if (open[j].hi > x.lo) open[k++] = open[j];
        open.resize(k);
        for (const Span& o : open) conflict = conflict || (o.call != x.call && (o.w || x.w));
        open.push_back(x);
    }
    if (!conflict) return 1;
    if (ndesc > MAX_LEVEL_CALLS) return 0;
    // where pieces start and end; most spans are those of other calls again
    std::vector<uintptr_t> cut;
    for (size_t i = 0; i < v.size(); i++) {
        if (i == 0 || v[i].lo != v[i - 1].lo) cut.push_back(v[i].lo);
        if (i == 0 || v[i].lo != v[i - 1].lo || v[i].hi != v[i - 1].hi) cut.push_back(v[i].hi);
    }
    std::sort(cut.begin(), cut.end());
    cut.erase(std::unique(cut.begin(), cut.end()), cut.end());
    struct Pieces {
        u32 first, end;
        int w;
    };
    std::vector<size_t> first(ndesc + 1, 0);   // of each call's spans
    for (const Span& x : v) first[x.call + 1]++;
    for (int i = 0; i < ndesc; i++) first[i + 1] += first[i];
    std::vector<size_t> next(first.begin(), first.end() - 1);
    std::vector<Pieces> spans(v.size());
    size_t lo = 0, pieces = 0;
    for (const Span& x : v) {
        while (cut[lo] != x.lo) lo++;
        const size_t hi = cut[lo + 1] == x.hi ? lo + 1 : std::lower_bound(cut.begin() + lo, cut.end(), x.hi) - cut.begin();
        pieces += hi - lo;
        spans[next[x.call]++] = {(u32)lo, (u32)hi, x.w};
    }
    if (pieces > MAX_LEVEL_PIECES) return 0;
    struct Piece {
        int written = 0, read = 0;   // level + 1 of its last writer and of its readers since
    };
    std::vector<Piece> piece(cut.size());
    int n = 1;
    for (int i = 0; i < ndesc; i++) {
        int l = 0;
        for (size_t k = first[i]; k < first[i + 1]; k++)
            for (u32 c = spans[k].first; c < spans[k].end; c++)
                l = std::max(l, spans[k].w ? std::max(piece[c].written, piece[c].read) : piece[c].written);
        for (int w : {0, 1})
            for (size_t k = first[i]; k < first[i + 1]; k++)
                for (u32 c = spans[k].first; spans[k].w == w && c < spans[k].end; c++) {
                    if (w) piece[c] = {l + 1, 0};
                    else piece[c].read = std::max(piece[c].read, l + 1);
                }
        level[i] = l;
        n = std::max(n, l + 1);
    }
    return n;
}

int launch(const void* kern, int grid, int threads, size_t smem, void* args, cudaStream_t st) {
    void* params[] = {args};
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CK(cudaLaunchKernelExC(&cfg, kern, params));
    g_launches++;
    return GPUMPI_OK;
}

// Kernel attributes belong to a device: once for each that plans are made on.
int spread_attributes() {
    static std::mutex mu;
    static std::vector<int> done;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (std::find(done.begin(), done.end(), dev) != done.end()) return GPUMPI_OK;
    for (const void* k : {(const void*)gpumpi_spread_kernel, (const void*)gpumpi_spread_params_kernel}) {
        CK(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
        CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SP_SMEM));
    }
    done.push_back(dev);
    return GPUMPI_OK;
}

// Independent tiles: any number of blocks, no cooperative launch, and blocks
// that may start before the launch before them has ended.
int launch_tiles(const void* kern, void* args, u32 ntiles, cudaStream_t st, bool overlap = true) {
    void* params[] = {args};
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(std::max(1u, std::min(ntiles, 1u << 30)));
    cfg.blockDim = dim3(SP_T);
    cfg.dynamicSmemBytes = SP_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    CK(cudaLaunchKernelExC(&cfg, kern, params));
    g_launches++;
    return GPUMPI_OK;
}

// Held while a plan's launches go to a stream: a plain launch that does not wait
// for those before it must follow its own plan's, not one that another thread
// put on the stream between two of them.  Streams share locks by their handles.
std::mutex& stream_lock(cudaStream_t st) {
    static std::mutex mu[64];
    const uintptr_t h = st == cudaStreamLegacy ? 0 : (uintptr_t)st;
    return mu[(h >> 4 ^ h >> 10) % 64];
}

int launch_spread(SpreadArgs* args, cudaStream_t st, bool overlap = true) {
    return launch_tiles((const void*)gpumpi_spread_kernel, args, args->ntiles, st, overlap);
}

}  // namespace

extern "C" int gpumpi_comm_create(int nranks, gpumpi_comm_t* out) {
    if (nranks <= 0 || !out) return GPUMPI_EINVAL;
    int rc = api_job();
    if (rc) return rc;
    const size_t n = (size_t)nranks;
    size_t off_cs = 0;
    size_t off_pub = 256;
    size_t off_flags = off_pub + ((sizeof(Pub) * n + 255) & ~(size_t)255);
    size_t off_h = off_flags + ((3 * sizeof(u64) * n + 255) & ~(size_t)255);
    size_t off_dc = off_h + ((sizeof(MPI_Comm_impl) * n + 255) & ~(size_t)255);
    size_t total = off_dc + 256;
    char* base = nullptr;
    CK(cudaMalloc(&base, total));
    CK(cudaMemset(base, 0, total));
    CommShared cs;
    memset(&cs, 0, sizeof(cs));
    cs.size = nranks;
    cs.ctx = 1;
    cs.members = nullptr;
    cs.pub = (Pub*)(base + off_pub);
    cs.arrive = (u64*)(base + off_flags);
    cs.mid = cs.arrive + n;
    cs.depart = cs.arrive + 2 * n;
    CK(cudaMemcpy(base + off_cs, &cs, sizeof(cs), cudaMemcpyHostToDevice));
    std::vector<MPI_Comm_impl> h(n);
    for (int r = 0; r < nranks; r++) {
        h[r].kind = 1;
        h[r].ctx = 1;
        h[r].size = nranks;
        h[r].rank = r;
        h[r].refcnt = 1;
        h[r].pad = 0;
        h[r].cs = (CommShared*)(base + off_cs);
        h[r].seq = 0;
    }
    CK(cudaMemcpy(base + off_h, h.data(), sizeof(MPI_Comm_impl) * n, cudaMemcpyHostToDevice));
    gpumpi_comm_s* c = new gpumpi_comm_s();
    c->n = nranks;
    c->base = base;
    c->hcomm.handles = (MPI_Comm_impl*)(base + off_h);
    c->hcomm.size = nranks;
    c->hcomm.pad = 0;
    c->dcomm = (DevComm*)(base + off_dc);
    CK(cudaMemcpy(c->dcomm, &c->hcomm, sizeof(DevComm), cudaMemcpyHostToDevice));
    *out = c;
    return GPUMPI_OK;
}

extern "C" int gpumpi_comm_destroy(gpumpi_comm_t c) {
    if (!c) return GPUMPI_EINVAL;
    cudaFree(c->base);
    delete c;
    return GPUMPI_OK;
}

extern "C" int gpumpi_comm_size(gpumpi_comm_t c, int* n) {
    if (!c || !n) return GPUMPI_EINVAL;
    *n = c->n;
    return GPUMPI_OK;
}

extern "C" int gpumpi_plan_create(const gpumpi_coll_desc* descs, int ndesc, int threads, int batched,
                                  gpumpi_plan_t* out) {
    return gpumpi_plan_create_ex(descs, ndesc, threads, batched, nullptr, out);
}

// upload: the stream whose work brings the tables, for a plan that is launched
// there only, first by plan_enqueue(p, st, true); null: they have arrived on return.
static int create_plan(const gpumpi_coll_desc* descs, int ndesc, int threads, int batched, const int* plain_threads,
                       const cudaStream_t* upload, gpumpi_plan_t* out) {
    if (!descs || ndesc <= 0 || !out) return GPUMPI_EINVAL;
    if (threads == 0) threads = 128;
    if (threads < 64 || threads > 1024 || threads % 32) return GPUMPI_EINVAL;
    for (int i = 0; plain_threads && i < ndesc; i++) {
        const int t = plain_threads[i];
        if (t != 0 && (t < 64 || t > 1024 || t % 32)) return GPUMPI_EINVAL;
    }
    int rc = api_job();
    if (rc) return rc;
    // communicators in order of first use; descriptors grouped by communicator, order kept
    std::vector<gpumpi_comm_t> comms;
    std::vector<int> cidx(ndesc);
    for (int i = 0; i < ndesc; i++) {
        const gpumpi_coll_desc& d = descs[i];
        if (!d.comm || esize_of(d.dtype) < 0 || d.op < 0 || d.op > GPUMPI_COLL_ALLGATHER) return GPUMPI_EINVAL;
        if ((d.op == GPUMPI_COLL_REDUCE || d.op == GPUMPI_COLL_ALLREDUCE) && (d.redop < 0 || d.redop > 3))
            return GPUMPI_EINVAL;
        if ((d.op == GPUMPI_COLL_BCAST || d.op == GPUMPI_COLL_REDUCE) && (d.root < 0 || d.root >= d.comm->n))
            return GPUMPI_EINVAL;
        if (d.algo < 0 || d.algo > 4) return GPUMPI_EINVAL;
        auto it = std::find(comms.begin(), comms.end(), d.comm);
        cidx[i] = (int)(it - comms.begin());
        if (it == comms.end()) comms.push_back(d.comm);
    }
    const int ncomm = (int)comms.size();
    std::vector<int> order(ndesc);
    for (int i = 0; i < ndesc; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cidx[a] < cidx[b]; });
    std::vector<int> comm_first(ncomm + 1, 0);
    for (int i = 0; i < ndesc; i++) comm_first[cidx[i] + 1]++;
    for (int c = 0; c < ncomm; c++) comm_first[c + 1] += comm_first[c];
    int total_slots = 0;
    for (auto* c : comms) total_slots += c->n;
    size_t ptrs = 0;
    for (int i = 0; i < ndesc; i++) ptrs += 2 * (size_t)descs[i].comm->n;
    // device layout: descs | comm_first | slot_comm | slot_rank | comms | per-desc comm_first pairs | pointers
    size_t off_desc = 0;
    size_t off_cf = off_desc + sizeof(DevDesc) * ndesc;
    size_t off_sc = (off_cf + sizeof(int) * (ncomm + 1) + 15) & ~(size_t)15;
    size_t off_sr = off_sc + sizeof(int) * total_slots;
    size_t off_cm = (off_sr + sizeof(int) * total_slots + 15) & ~(size_t)15;
    size_t off_pp = off_cm + sizeof(DevComm) * ncomm;
    size_t off_pc = (off_pp + sizeof(int) * 2 * ndesc + 15) & ~(size_t)15;
    size_t off_ptr = off_pc + sizeof(DevComm) * ndesc;
    size_t off_pubt = (off_ptr + sizeof(void*) * ptrs + 63) & ~(size_t)63;   // Pub tables, one entry per rank
    const size_t off_sp = off_pubt + sizeof(Pub) * (ptrs / 2);   // SpreadCalls, then their address tables
    // the spread form: the whole batched launch, or each plain launch it covers
    std::unique_ptr<gpumpi_plan_s> p(new gpumpi_plan_s());   // gone with its memory on any error below
    std::vector<int> level;
    const int nlevels = plan_levels(descs, ndesc, level);
    p->independent = nlevels == 1;
    std::vector<SpreadBuilder> spread(batched ? 1 : ndesc);
    std::vector<char> overlap(ndesc, 0);
    p->plain_spread.assign(ndesc, 0);
    p->plain_tiles.resize(ndesc);
    auto covers = [&](int i) { return SpreadBuilder::covers(descs[i], descs[i].comm->n, esize_of(descs[i].dtype)); };
    if (batched) {
        std::vector<SpreadLoad> load(nlevels);
        p->batch_spread = nlevels > 0;
        for (int i = 0; i < ndesc && p->batch_spread; i++) {
            p->batch_spread = covers(i);
            load[level[i]].count(descs[i], descs[i].comm->n, esize_of(descs[i].dtype));
        }
        for (int l = 0; l < nlevels && p->batch_spread; l++) {
            for (int i = 0; i < ndesc; i++)
                if (level[i] == l) spread[0].add(descs[i], descs[i].comm->n, esize_of(descs[i].dtype), load[l]);
            spread[0].end_level();
        }
    } else {
        for (int k = 0; k < ndesc; k++) {
            const int i = order[k];
            p->plain_spread[k] = covers(i);
            if (!p->plain_spread[k]) continue;
            SpreadLoad load;
            load.count(descs[i], descs[i].comm->n, esize_of(descs[i].dtype));
            spread[k].add(descs[i], descs[i].comm->n, esize_of(descs[i].dtype), load);
            spread[k].end_level();
        }
        // launch k need not wait for those from k0, the last that does, to k - 1
        // when they are of one level: calls of a level touch disjoint memory
        int k0 = 0;
        for (int k = 0; k < ndesc; k++) {
            overlap[k] = k > k0 && nlevels > 0 && p->plain_spread[k] && p->plain_spread[k - 1] &&
                         level[order[k]] == level[order[k0]];
            if (!overlap[k]) k0 = k;
        }
    }
    size_t total = off_sp;
    for (const SpreadBuilder& b : spread) total += b.bytes() + 64;
    // Room for the tile lists of a host-buffer call's groups (make_pipe fills it in
    // with the first of those calls, which therefore allocates no device memory).
    if (p->batch_spread && nlevels == 1 && ndesc > 1) {
        size_t moved = 0, in, out, room = 0;
        for (int i = 0; i < ndesc; i++) {
            moved += host_bytes(descs[i], descs[i].comm->n, &in, &out);
            room += SpreadBuilder::max_bytes(descs[i].comm->n);
        }
        if (moved >= PIPE_MIN_BYTES) p->pipe_bytes = room + (PIPE_GROUPS + 1) * 64;
    }
    const size_t off_pipe = (total + 63) & ~(size_t)63;
    CK(cudaMalloc(&p->base, off_pipe + p->pipe_bytes));
    char* base = p->base;
    p->pipe_base = base + off_pipe;
    std::vector<char> h(total, 0);
    DevDesc* hd = (DevDesc*)(h.data() + off_desc);
    void** hp = (void**)(h.data() + off_ptr);
    Pub* hpub = (Pub*)(h.data() + off_pubt);
    size_t pk = 0, pubk = 0;
    p->descs.assign(descs, descs + ndesc);
    p->sb.resize(ndesc);
    p->rb.resize(ndesc);
    for (int k = 0; k < ndesc; k++) {
        const int i = order[k];
        const gpumpi_coll_desc& d = descs[i];
        const int P = d.comm->n;
        DevDesc& x = hd[k];
        x.op = d.op;
        x.dtype = d.dtype;
        x.redop = d.redop;
        x.root = d.root;
        x.count = d.count;
        x.comm = cidx[i];
        x.esize = esize_of(d.dtype);
        x.algo = d.algo;
        x.sync = d.sync ? 1 : 0;
        x.sbufs = (void**)(base + off_ptr + sizeof(void*) * pk);
        for (int r = 0; r < P; r++) hp[pk++] = d.sendbufs ? d.sendbufs[r] : nullptr;
        x.rbufs = (void**)(base + off_ptr + sizeof(void*) * pk);
        for (int r = 0; r < P; r++) hp[pk++] = d.recvbufs ? d.recvbufs[r] : nullptr;
        p->sb[i].assign(hp + pk - 2 * P, hp + pk - P);
        p->rb[i].assign(hp + pk - P, hp + pk);
        x.pub = (const Pub*)(base + off_pubt) + pubk;
        for (int r = 0; r < P; r++, pubk++) {
            Pub& e = hpub[pubk];
            e.rbuf = d.recvbufs ? d.recvbufs[r] : nullptr;
            e.sbuf = d.sendbufs ? d.sendbufs[r] : e.rbuf;
            e.a0 = (long long)d.count;
            e.a1 = x.esize;
        }
    }
    memcpy(h.data() + off_cf, comm_first.data(), sizeof(int) * (ncomm + 1));
    int* sc = (int*)(h.data() + off_sc);
    int* sr = (int*)(h.data() + off_sr);
    int s = 0;
    for (int c = 0; c < ncomm; c++)
        for (int r = 0; r < comms[c]->n; r++) {
            sc[s] = c;
            sr[s] = r;
            s++;
        }
    DevComm* hc = (DevComm*)(h.data() + off_cm);
    for (int c = 0; c < ncomm; c++) hc[c] = comms[c]->hcomm;
    // plain launches: each descriptor alone, its own communicator at index 0
    int* pp = (int*)(h.data() + off_pp);
    DevComm* pc = (DevComm*)(h.data() + off_pc);
    for (int k = 0; k < ndesc; k++) {
        pp[2 * k] = 0;
        pp[2 * k + 1] = 1;
        pc[k] = comms[hd[k].comm]->hcomm;
    }
    size_t at = off_sp;
    for (size_t k = 0; k < spread.size(); k++) {
        at = (at + 63) & ~(size_t)63;
        if (batched) p->batch_tiles.resize(spread[k].levels.size());
        SpreadArgs* a = batched ? p->batch_tiles.data() : &p->plain_tiles[k];
        spread[k].image(h.data() + at, base + at, a);
        for (size_t l = 0; l < spread[k].levels.size(); l++) {
            a[l].job = g_api.djob;
            a[l].overlap = !batched && overlap[k];
        }
        at += spread[k].bytes();
    }
    if (upload) {
        p->image = std::move(h);
        CK(cudaMemcpyAsync(base, p->image.data(), total, cudaMemcpyHostToDevice, *upload));
    } else {
        CK(cudaMemcpy(base, h.data(), total, cudaMemcpyHostToDevice));
        // a copy from pageable memory may return before it has arrived, and launches on
        // any stream read the tables before they wait for anything
        CK(cudaStreamSynchronize(cudaStreamLegacy));
    }
    p->ndesc = ndesc;
    p->ncomm = ncomm;
    p->batched = batched;
    p->threads = threads;
    p->smem = rank_smem_bytes(0);
    p->total_slots = total_slots;
    p->batch_args.job = g_api.djob;
    p->batch_args.descs = (const DevDesc*)(base + off_desc);
    p->batch_args.comm_first = (const int*)(base + off_cf);
    p->batch_args.slot_comm = (const int*)(base + off_sc);
    p->batch_args.slot_rank = (const int*)(base + off_sr);
    p->batch_args.comms = (const DevComm*)(base + off_cm);
    p->batch_args.ordered = p->independent;
    p->batch_args.pad = 0;
    p->plain_args.resize(ndesc);
    p->plain_grid.resize(ndesc);
    p->plain_threads.resize(ndesc);
    for (int k = 0; k < ndesc; k++) {
        const int t = plain_threads ? plain_threads[order[k]] : 0;
        p->plain_threads[k] = t ? t : threads;
        PlanArgs& a = p->plain_args[k];
        a.job = g_api.djob;
        a.descs = (const DevDesc*)(base + off_desc) + k;
        a.comm_first = (const int*)(base + off_pp) + 2 * k;
        a.slot_comm = nullptr;
        a.slot_rank = nullptr;
        a.comms = (const DevComm*)(base + off_pc) + k;
        a.ordered = hd[k].op != GPUMPI_COLL_BARRIER;   // one call per launch: always launch-ordered
        a.pad = 0;
        p->plain_op.push_back(hd[k].op);
        p->plain_grid[k] = comms[hd[k].comm]->n;
    }
    // co-residency: every rank block of one launch must fit on the GPU at once
    int per = 0, sms = 0, dev = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    p->plain_smem.assign(ndesc, rank_smem_bytes(0));
    for (int k = 0; k <= ndesc; k++) {
        // k < ndesc: each plain launch at its own thread count; k == ndesc: the batched launch
        if (k < ndesc && batched) continue;
        if (k == ndesc && !batched) break;
        const int t = k < ndesc ? p->plain_threads[k] : threads;
        const int need = k < ndesc ? p->plain_grid[k] : total_slots;
        const size_t smem = pick_rank_smem((const void*)gpumpi_plan_kernel, t, need);
        if (k < ndesc) p->plain_smem[k] = smem;
        else p->smem = smem;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)gpumpi_plan_kernel, t, smem));
        if ((long long)per * sms < need) {
            char m[200];
            snprintf(m, sizeof(m), "%d rank blocks of %d threads cannot be co-resident (max %d)", need, t,
                     per * sms);
            set_last_error(m);
            return GPUMPI_ENORES;
        }
    }
    *out = p.release();
    return GPUMPI_OK;
}

extern "C" int gpumpi_plan_create_ex(const gpumpi_coll_desc* descs, int ndesc, int threads, int batched,
                                     const int* plain_threads, gpumpi_plan_t* out) {
    return create_plan(descs, ndesc, threads, batched, plain_threads, nullptr, out);
}

// first: the plan's tables arrive on `st` just before, so its first launch may not
// start ahead of that; the later ones start when the first has.
static int plan_enqueue(gpumpi_plan_t p, cudaStream_t st, bool first = false) {
    const void* k = (const void*)gpumpi_plan_kernel;
    std::lock_guard<std::mutex> lock(stream_lock(st));
    if (p->batched) {
        if (p->batch_spread && p->sync_mode == 0) {
            // A launch for each level.  One launch with a barrier of all its blocks
            // between two levels needs them all on the GPU at once, so it waits for
            // every kernel that holds some of it, and is slower: five dependent calls
            // of 4 ranks of 200 FP64 22.7 us, so 11.6; of 48 of 20000 38.4, 28.3; of 200
            // of 131072 517, 463; 400 calls of 8 ranks of one element 1481, 824.
            for (SpreadArgs& a : p->batch_tiles) {
                int rc = launch_spread(&a, st, !first);
                if (rc) return rc;
                first = false;
            }
            return GPUMPI_OK;
        }
        return launch(k, p->total_slots, p->threads, p->smem, &p->batch_args, st);
    }
    for (int i = 0; i < p->ndesc; i++) {
        int rc = p->plain_spread[i] && p->plain_args[i].ordered
                     ? launch_spread(&p->plain_tiles[i], st, !first)
                     : launch(k, p->plain_grid[i], p->plain_threads[i], p->plain_smem[i], &p->plain_args[i], st);
        if (rc) return rc;
        first = false;
    }
    return GPUMPI_OK;
}

// One launch of independent tiles, which may start while the launch before it ends.
static bool one_launch(gpumpi_plan_t p) {
    return p->batched && p->batch_spread && p->sync_mode == 0 && p->batch_tiles.size() == 1;
}

// True when everything that `st` was given has run.  By the driver's function,
// which leaves the runtime's last error alone, in the relaxed mode, which no
// capture of another thread minds; a stream under capture is not asked.
static bool stream_idle(cudaStream_t st) {
    typedef int (*QueryFn)(cudaStream_t);
    static QueryFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuStreamQuery", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (QueryFn)f;
        cudaGetLastError();
        return (QueryFn) nullptr;
    }();
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusActive;
    if (!fn || cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone)
        return false;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return false;
    const bool idle = fn(st) == 0;
    cudaThreadExchangeStreamCaptureMode(&mode);
    return idle;
}

extern "C" int gpumpi_plan_launch(gpumpi_plan_t p, void* stream) {
    if (!p) return GPUMPI_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    // A graph cannot overlap the launch before it, so that of a single launch of
    // tiles is for a stream that has nothing else to do (the 16-communicator batch at
    // 1 element per rank, graph / launched: with a wait after each 22.0 / 23.4 us, back
    // to back 16.4 / 13.1).
    if (p->exec && (!one_launch(p) || stream_idle(st))) {
        CK(cudaGraphLaunch(p->exec, st));
        g_launches += !p->batched ? p->ndesc : p->batch_spread && p->sync_mode == 0 ? p->batch_tiles.size() : 1;
        return GPUMPI_OK;
    }
    return plan_enqueue(p, st);
}

extern "C" int gpumpi_plan_set_sync(gpumpi_plan_t p, int mode) {
    if (!p || mode < 0 || mode > 1) return GPUMPI_EINVAL;
    p->sync_mode = mode;
    p->batch_args.ordered = mode == 0 && p->independent;
    for (int k = 0; k < p->ndesc; k++)
        p->plain_args[k].ordered = mode == 0 && p->plain_op[k] != GPUMPI_COLL_BARRIER;
    // a captured graph holds the old launch arguments: launch eagerly until captured again
    if (p->exec) cudaGraphExecDestroy(p->exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    p->exec = nullptr;
    p->graph = nullptr;
    return GPUMPI_OK;
}

extern "C" int gpumpi_plan_launch_ordered(gpumpi_plan_t p) {
    if (!p) return 0;
    return p->batched ? p->batch_args.ordered : (p->sync_mode == 0);
}

extern "C" int gpumpi_plan_capture(gpumpi_plan_t p, void* stream) {
    if (!p) return GPUMPI_EINVAL;
    (void)stream;   // captured on a private stream; replays go to the stream given to gpumpi_plan_launch
    cudaStream_t cap;
    CK(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    CK(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    unsigned long long before = g_launches;
    int rc = plan_enqueue(p, cap);
    g_launches = before;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(cap, &g);
    if (!rc && e == cudaSuccess) e = cudaGraphInstantiate(&p->exec, g, 0);
    // its first replay need not bring it to the device (31.8 us launched, 33.3 without)
    if (!rc && e == cudaSuccess && (cudaGraphUpload(p->exec, cap) != cudaSuccess || cudaStreamSynchronize(cap) != cudaSuccess))
        cudaGetLastError();
    cudaStreamDestroy(cap);
    if (rc) return rc;
    CK(e);
    p->graph = g;
    return GPUMPI_OK;
}

// Host-buffer path: copy every rank's send data from host memory, run the
// plan, copy every rank's result back.  host_send/host_recv hold, for each
// descriptor in the order given to gpumpi_plan_create, one host pointer per
// rank (nullptr = skip).
namespace {

// Copies of one direction, merged while both sides continue where the
// previous copy ended, within one descriptor, the device side inside one
// allocation (cuMemGetAddressRange, fetched through the runtime) and the host
// side of one memory type; rank buffers carved from one allocation on each
// side become one cudaMemcpyAsync.
typedef int (*AddrRangeFn)(unsigned long long* base, size_t* size, unsigned long long ptr);

AddrRangeFn addr_range() {
    static AddrRangeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (AddrRangeFn)f;
        cudaGetLastError();
        return (AddrRangeFn) nullptr;
    }();
    return fn;
}

// End of the pinned allocation or registration that holds host address p, 0
// where the driver does not say.
uintptr_t pinned_end(const void* p) {
    typedef int (*AttrFn)(void* data, int attribute, unsigned long long ptr);
    static AttrFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (AttrFn)f;
        cudaGetLastError();
        return (AttrFn) nullptr;
    }();
    constexpr int RANGE_START = 11, RANGE_SIZE = 12;   // CU_POINTER_ATTRIBUTE_RANGE_*
    unsigned long long start = 0;
    size_t size = 0;
    if (!fn || fn(&start, RANGE_START, (uintptr_t)p) || fn(&size, RANGE_SIZE, (uintptr_t)p)) return 0;
    return (uintptr_t)p - start < size ? (uintptr_t)(start + size) : 0;
}

int host_kind(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return (int)a.type;
}

struct CopyRun {
    int desc;
    char* dst;
    const char* src;
    size_t n;
    unsigned long long dev_end;   // end of the device allocation of the run (0: unknown)
    int hkind;                    // memory type of its host side (-1: unknown)
    uintptr_t host_end;           // end of the host side's allocation (0: unknown)
};

void add_copy(std::vector<CopyRun>& runs, int desc, void* d, const void* s, size_t len, bool to_dev) {
    const unsigned long long dptr = (unsigned long long)(to_dev ? (uintptr_t)d : (uintptr_t)s);
    const void* hptr = to_dev ? s : (const void*)d;
    if (!runs.empty()) {
        CopyRun& r = runs.back();
        if (desc == r.desc && (char*)d == r.dst + r.n && (const char*)s == r.src + r.n && dptr + len <= r.dev_end &&
            r.hkind >= 0 && ((uintptr_t)hptr + len <= r.host_end || host_kind(hptr) == r.hkind)) {
            r.n += len;
            return;
        }
    }
    CopyRun r = {desc, (char*)d, (const char*)s, len, 0, -1, 0};
    unsigned long long base = 0;
    size_t size = 0;
    AddrRangeFn f = addr_range();
    if (f && f(&base, &size, dptr) == 0) {
        r.dev_end = base + size;
        r.hkind = host_kind(hptr);
        if (r.hkind == (int)cudaMemoryTypeHost) r.host_end = pinned_end(hptr);
    }
    runs.push_back(r);
}

int enqueue_copies(const std::vector<CopyRun>& runs, int desc, cudaMemcpyKind kind, cudaStream_t st) {
    for (const CopyRun& r : runs)
        if (desc < 0 || r.desc == desc) CK(cudaMemcpyAsync(r.dst, r.src, r.n, kind, st));
    return GPUMPI_OK;
}

// The groups of a plan, calls with the most output for their input first, so
// that the way back is busy from the start.  On an error the pipe is as before
// and the next call tries again.
int make_pipe(gpumpi_plan_t p, HostPipe& pipe) {
    if (!p->pipe_bytes) {
        pipe.state = HostPipe::NONE;
        return GPUMPI_OK;
    }
    // the caller's address tables may be gone: the plan's own copies
    std::vector<gpumpi_coll_desc> descs(p->descs);
    for (int i = 0; i < p->ndesc; i++) {
        if (descs[i].sendbufs) descs[i].sendbufs = p->sb[i].data();
        descs[i].recvbufs = p->rb[i].data();
    }
    std::vector<int> level;
    if (plan_levels(descs.data(), p->ndesc, level, true) != 1) {
        pipe.state = HostPipe::NONE;
        return GPUMPI_OK;
    }
    std::vector<size_t> in(p->ndesc), out(p->ndesc);
    std::vector<int> order(p->ndesc);
    size_t total = 0;
    for (int i = 0; i < p->ndesc; i++) {
        total += host_bytes(p->descs[i], p->descs[i].comm->n, &in[i], &out[i]);
        order[i] = i;
    }
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return in[a] / (out[a] + 1.0) < in[b] / (out[b] + 1.0); });
    size_t held = 0;
    for (int i : order) {
        if (held == 0) pipe.groups.emplace_back();
        pipe.groups.back().push_back(i);
        held += in[i] + out[i];
        if (held >= total / PIPE_GROUPS) held = 0;
    }
    if (pipe.groups.size() < 2) {
        pipe.state = HostPipe::NONE;
        return GPUMPI_OK;
    }
    std::vector<SpreadBuilder> tiles(pipe.groups.size());
    size_t bytes = 0;
    for (size_t g = 0; g < pipe.groups.size(); g++) {
        SpreadLoad load;
        for (int i : pipe.groups[g]) load.count(descs[i], descs[i].comm->n, esize_of(descs[i].dtype));
        for (int i : pipe.groups[g]) tiles[g].add(descs[i], descs[i].comm->n, esize_of(descs[i].dtype), load);
        tiles[g].end_level();
        bytes += (tiles[g].bytes() + 63) & ~(size_t)63;
    }
    if (bytes > p->pipe_bytes) {   // not reached: max_bytes() bounds every call
        pipe.state = HostPipe::NONE;
        return GPUMPI_OK;
    }
    pipe.image.resize(bytes);
    pipe.tiles.resize(tiles.size());
    size_t at = 0;
    for (size_t g = 0; g < tiles.size(); g++) {
        tiles[g].image(pipe.image.data() + at, p->pipe_base + at, &pipe.tiles[g]);
        pipe.tiles[g].job = g_api.djob;
        at += (tiles[g].bytes() + 63) & ~(size_t)63;
    }
    CK(cudaStreamCreateWithFlags(&pipe.in, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&pipe.out, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&pipe.begin, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&pipe.end, cudaEventDisableTiming));
    for (size_t g = 0; g < tiles.size(); g++) {
        cudaEvent_t e;
        CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        pipe.arrived.push_back(e);
        CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        pipe.ran.push_back(e);
    }
    // Ahead of every group's inputs on the stream that brings them, so a launch on
    // any stream that waits for its inputs waits for its tiles too.
    CK(cudaMemcpyAsync(p->pipe_base, pipe.image.data(), bytes, cudaMemcpyHostToDevice, pipe.in));
    pipe.state = HostPipe::READY;
    return GPUMPI_OK;
}

// Every copy between pinned host memory and the device, and no host byte both
// read and written: then the order of the copies in and out does not matter.
bool host_disjoint(const std::vector<CopyRun>& in, const std::vector<CopyRun>& out) {
    struct Span {
        uintptr_t lo, hi;
        bool w;
    };
    std::vector<Span> v;
    for (const CopyRun& r : in) {
        if (r.hkind != (int)cudaMemoryTypeHost) return false;
        v.push_back({(uintptr_t)r.src, (uintptr_t)r.src + r.n, false});
    }
    for (const CopyRun& r : out) {
        if (r.hkind != (int)cudaMemoryTypeHost) return false;
        v.push_back({(uintptr_t)r.dst, (uintptr_t)r.dst + r.n, true});
    }
    std::sort(v.begin(), v.end(), [](const Span& a, const Span& b) { return a.lo < b.lo; });
    uintptr_t end[2] = {0, 0};   // of the spans so far: read, written
    for (const Span& s : v) {
        if (s.lo < end[1] || (s.w && s.lo < end[0])) return false;
        end[s.w] = std::max(end[s.w], s.hi);
    }
    return true;
}

int pipe_groups(HostPipe& pipe, const std::vector<CopyRun>& in, const std::vector<CopyRun>& out, cudaStream_t st) {
    CK(cudaEventRecord(pipe.begin, st));
    CK(cudaStreamWaitEvent(pipe.in, pipe.begin, 0));
    for (size_t g = 0; g < pipe.groups.size(); g++) {
        int rc = GPUMPI_OK;
        for (int d : pipe.groups[g])
            if (!rc) rc = enqueue_copies(in, d, cudaMemcpyHostToDevice, pipe.in);
        if (rc) return rc;
        CK(cudaEventRecord(pipe.arrived[g], pipe.in));
        CK(cudaStreamWaitEvent(st, pipe.arrived[g], 0));
        {
            std::lock_guard<std::mutex> turn(stream_lock(st));
            rc = launch_tiles((const void*)gpumpi_spread_kernel, &pipe.tiles[g], pipe.tiles[g].ntiles, st, false);
        }
        if (rc) return rc;
        CK(cudaEventRecord(pipe.ran[g], st));
        CK(cudaStreamWaitEvent(pipe.out, pipe.ran[g], 0));
        for (int d : pipe.groups[g])
            if (!rc) rc = enqueue_copies(out, d, cudaMemcpyDeviceToHost, pipe.out);
        if (rc) return rc;
    }
    CK(cudaEventRecord(pipe.end, pipe.out));
    CK(cudaStreamWaitEvent(st, pipe.end, 0));
    return GPUMPI_OK;
}

int run_pipe(HostPipe& pipe, const std::vector<CopyRun>& in, const std::vector<CopyRun>& out, cudaStream_t st) {
    const int rc = pipe_groups(pipe, in, out, st);
    if (!rc) return rc;
    // copies that are under way still use the caller's memory: the caller, who
    // knows of `st` only, waits for them there, or here if that cannot be had
    for (cudaStream_t s : {pipe.in, pipe.out})
        if (cudaEventRecord(pipe.end, s) != cudaSuccess || cudaStreamWaitEvent(st, pipe.end, 0) != cudaSuccess) {
            cudaGetLastError();
            cudaStreamSynchronize(s);
        }
    return rc;
}

// One after another on one stream.
int host_enqueue(gpumpi_plan_t p, const std::vector<CopyRun>& in, const std::vector<CopyRun>& out, cudaStream_t st) {
    int rc = enqueue_copies(in, -1, cudaMemcpyHostToDevice, st);
    if (!rc) rc = gpumpi_plan_launch(p, st);
    if (!rc) rc = enqueue_copies(out, -1, cudaMemcpyDeviceToHost, st);
    return rc;
}

}  // namespace

extern "C" int gpumpi_plan_run_host(gpumpi_plan_t p, void* const* host_send, void* const* host_recv,
                                    void* stream, uint64_t* h2d_bytes, uint64_t* d2h_bytes) {
    if (!p) return GPUMPI_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    size_t k = 0, bi = 0, bo = 0;
    std::vector<CopyRun> to_dev, to_host;
    for (int d = 0; d < p->ndesc; d++) {
        const int P = p->descs[d].comm->n;
        const int op = p->descs[d].op, root = p->descs[d].root;
        size_t in, out;
        desc_bytes(p->descs[d], P, &in, &out);
        for (int r = 0; r < P; r++, k++) {
            void* dst = op == GPUMPI_COLL_BCAST ? p->rb[d][r] : p->sb[d][r];
            if ((op != GPUMPI_COLL_BCAST || r == root) && host_send && host_send[k] && dst && in) {
                add_copy(to_dev, d, dst, host_send[k], in, true);
                bi += in;
            }
            if ((op != GPUMPI_COLL_REDUCE || r == root) && host_recv && host_recv[k] && p->rb[d][r] && out) {
                add_copy(to_host, d, host_recv[k], p->rb[d][r], out, false);
                bo += out;
            }
        }
    }
    if (h2d_bytes) *h2d_bytes = bi;
    if (d2h_bytes) *d2h_bytes = bo;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(st, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) return host_enqueue(p, to_dev, to_host, st);
    // The calls of a plan share its device buffers: each starts when the one
    // before it has ended, whatever their streams.
    std::lock_guard<std::mutex> lock(p->pipe_mu);
    if (!p->host_done) CK(cudaEventCreateWithFlags(&p->host_done, cudaEventDisableTiming));
    else CK(cudaStreamWaitEvent(st, p->host_done, 0));
    // Copies in, launches and copies out of groups of calls on three streams: the
    // link carries both directions at once (three communicators of 128, 88 and 40
    // ranks, 2^14 elements per rank: 1438 us one after another, 1010 us so; alone,
    // with a wait, 1.80 and 1.31 ms).
    bool piped = bi + bo >= PIPE_MIN_BYTES && p->sync_mode == 0;
    if (piped && p->pipe.state == HostPipe::NEW && make_pipe(p, p->pipe)) {
        cudaGetLastError();
        p->pipe.drop();
    }
    piped = piped && p->pipe.state == HostPipe::READY && host_disjoint(to_dev, to_host);
    const int rc = piped ? run_pipe(p->pipe, to_dev, to_host, st) : host_enqueue(p, to_dev, to_host, st);
    if (rc) cudaEventRecord(p->host_done, st);   // the message is that of rc
    else CK(cudaEventRecord(p->host_done, st));
    return rc;
}

extern "C" int gpumpi_plan_destroy(gpumpi_plan_t p) {
    if (!p) return GPUMPI_EINVAL;
    delete p;
    return GPUMPI_OK;
}

extern "C" int gpumpi_api_status(char* msg, int len);
static int one_shot(const gpumpi_coll_desc* descs, int ndesc, int threads, void* stream, int batched) {
    // The tables come in the stream's order: a wait for them alone would be 7 us of a
    // single call's 43 (rank blocks, which did without, 34).
    gpumpi_plan_t p = nullptr;
    cudaStream_t st = (cudaStream_t)stream;
    int rc = create_plan(descs, ndesc, threads, batched, nullptr, &st, &p);
    if (rc) return rc;
    rc = plan_enqueue(p, st, true);
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    gpumpi_plan_destroy(p);
    if (rc) return rc;
    if (e != cudaSuccess) return GPUMPI_ECUDA;
    return gpumpi_api_status(nullptr, 0);
}

extern "C" int gpumpi_coll_plain(const gpumpi_coll_desc* descs, int ndesc, int threads, void* stream) {
    return one_shot(descs, ndesc, threads, stream, 0);
}

extern "C" int gpumpi_coll_batched(const gpumpi_coll_desc* descs, int ndesc, int threads, void* stream) {
    return one_shot(descs, ndesc, threads, stream, 1);
}

// Error state of the collective API's device job; clears it.
extern "C" int gpumpi_api_status(char* msg, int len) {
    if (!g_api.djob) return GPUMPI_OK;
    int st[16];
    CK(cudaMemcpy(st, g_api.status, sizeof(st), cudaMemcpyDeviceToHost));
    if (st[1] == 0) return GPUMPI_OK;
    char m[256];
    CK(cudaMemcpy(m, g_api.err, sizeof(m), cudaMemcpyDeviceToHost));
    m[255] = 0;
    if (msg && len > 0) snprintf(msg, len, "error %d on rank %d: %s", st[1], st[2], m);
    char full[320];
    snprintf(full, sizeof(full), "collective job error %d on rank %d: %s", st[1], st[2], m);
    set_last_error(full);
    CK(cudaMemset(g_api.status, 0, sizeof(st)));
    return GPUMPI_EJOB;
}

extern "C" uint64_t gpumpi_kernel_launches(void) { return g_launches; }

// ------------------------------------------------------------------ allocation-free allreduce
// Some callers may not allocate device memory on their call path: a serving
// loop that reserved all of HBM when it started, a host thread running under
// a pooled allocator's fixed budget, or code that must not block the device
// (cudaMalloc and cudaFree can synchronise it).  gpumpi_allreduce_noalloc
// serves them: it runs the same allreduce schedule as the plan kernel, but
// its synchronisation state (communicator tables, flags, per-rank handles,
// error words) lives in the fixed array below instead of cudaMalloc'd memory.
//
// Calls of the arithmetic types run as independent tiles instead, with their
// descriptors among the kernel's parameters, and do not touch the array.
//
// The array is a file-scope device variable, so every GPU that loads this
// library holds it until the process exits, and every call shares it: each
// call rewrites the part it uses (clearing the flags), and calls whose
// kernels overlap on the GPU race on it.  Host code may not use the array's
// name as a device address; the entry point looks the address up with
// cudaGetSymbolAddress the first time it runs on a device (with that device
// current), so that first call should come before any stream capture.
namespace {

constexpr int NOALLOC_MAX_RANKS = 256;
constexpr size_t NOALLOC_SCRATCH_BYTES = 64 * 1024;

static __device__ __align__(256) unsigned char gm_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

struct NoallocLayout {
    size_t job, status, err, cs, pub, flags, handles, dcomm, desc, first, ptrs, total;
};

constexpr size_t noalloc_take(size_t& o, size_t bytes) {
    o = (o + 255) & ~(size_t)255;
    const size_t at = o;
    o += bytes;
    return at;
}

constexpr NoallocLayout noalloc_layout(int n) {
    NoallocLayout L{};
    size_t o = 0;
    L.job = noalloc_take(o, sizeof(Job));
    L.status = noalloc_take(o, sizeof(int) * 16);
    L.err = noalloc_take(o, 256);
    L.cs = noalloc_take(o, sizeof(CommShared));
    L.pub = noalloc_take(o, sizeof(Pub) * (size_t)n);
    L.flags = noalloc_take(o, sizeof(u64) * 3 * (size_t)n);
    L.handles = noalloc_take(o, sizeof(MPI_Comm_impl) * (size_t)n);
    L.dcomm = noalloc_take(o, sizeof(DevComm));
    L.desc = noalloc_take(o, sizeof(DevDesc));
    L.first = noalloc_take(o, sizeof(int) * 2);
    L.ptrs = noalloc_take(o, sizeof(void*) * 2 * (size_t)n);
    L.total = noalloc_take(o, 0);
    return L;
}

// The layout grows with the rank count; the largest one must fit the array
// (a larger Job, Pub or communicator record fails the build here instead of
// overflowing the array at run time).
static_assert(noalloc_layout(NOALLOC_MAX_RANKS).total <= NOALLOC_SCRATCH_BYTES,
              "allocation-free allreduce: scratch array too small for NOALLOC_MAX_RANKS");

std::mutex g_noalloc_mu;
void* g_noalloc_dev_ptr[64];                                    // per device, looked up once
unsigned char g_noalloc_image[NOALLOC_SCRATCH_BYTES];           // host image of the used prefix

}  // namespace

// See include/gpumpi.h.  Synchronises `stream`; returns 0 or an error code.
extern "C" int gpumpi_allreduce_noalloc(void* const* sendbufs, void* const* recvbufs, int nranks,
                                        uint64_t count, int dtype, int redop, int threads_per_rank,
                                        void* stream) {
    if (nranks < 1 || nranks > NOALLOC_MAX_RANKS) {
        char m[160];
        snprintf(m, sizeof(m), "gpumpi_allreduce_noalloc: %d ranks requested, the fixed scratch holds at most %d",
                 nranks, NOALLOC_MAX_RANKS);
        set_last_error(m);
        return GPUMPI_EINVAL;
    }
    const int es = esize_of(dtype);
    if (!sendbufs || !recvbufs || es < 0 || redop < 0 || redop > 3) {
        set_last_error("gpumpi_allreduce_noalloc: bad buffers, datatype or operator");
        return GPUMPI_EINVAL;
    }
    if (threads_per_rank == 0) threads_per_rank = 128;
    if (threads_per_rank < 64 || threads_per_rank > 1024 || threads_per_rank % 32) {
        set_last_error("gpumpi_allreduce_noalloc: threads_per_rank must be a multiple of 32 in [64, 1024]");
        return GPUMPI_EINVAL;
    }
    for (int r = 0; r < nranks; r++)
        if (!sendbufs[r] || !recvbufs[r]) {
            set_last_error("gpumpi_allreduce_noalloc: a send or receive buffer is NULL");
            return GPUMPI_EINVAL;
        }
    std::unique_lock<std::mutex> lock(g_noalloc_mu);
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_last_error("gpumpi_allreduce_noalloc: device ordinal above 63");
        return GPUMPI_EINVAL;
    }
    if (!g_noalloc_dev_ptr[dev]) {
        int rc = spread_attributes();
        if (rc) return rc;
        void* p = nullptr;
        CK(cudaGetSymbolAddress(&p, gm_noalloc_scratch));
        g_noalloc_dev_ptr[dev] = p;
    }
    char* base = (char*)g_noalloc_dev_ptr[dev];
    const NoallocLayout L = noalloc_layout(nranks);
    if (L.total > NOALLOC_SCRATCH_BYTES) {   // unreachable while the static_assert holds
        set_last_error("gpumpi_allreduce_noalloc: layout exceeds the scratch array");
        return GPUMPI_EINVAL;
    }
    const size_t smem = sizeof(BlockCtx) + 64;
    int per = 0, sms = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)gpumpi_plan_kernel, threads_per_rank, smem));
    if ((long long)per * sms < nranks) {
        set_last_error("gpumpi_allreduce_noalloc: rank blocks cannot all be resident");
        return GPUMPI_ENORES;
    }
    cudaStream_t st = (cudaStream_t)stream;
    gpumpi_coll_desc call;
    memset(&call, 0, sizeof(call));
    call.op = GPUMPI_COLL_ALLREDUCE;
    call.dtype = dtype;
    call.redop = redop;
    call.count = count;
    call.sendbufs = sendbufs;
    call.recvbufs = recvbufs;
    if (SpreadBuilder::covers(call, nranks, es)) {
        // Independent tiles with all they need among the kernel's parameters: no
        // device memory, no copies, nothing shared between calls, and no wait
        // that could fail (32 ranks of 4096 FP64 elements: 63 us by the rank
        // form below with its image copied in and its status out, 17 us so).
        SpreadBuilder tiles;
        SpreadParams params;
        SpreadLoad load;
        load.count(call, nranks, es);
        tiles.add(call, nranks, es, load);
        tiles.end_level();
        if (tiles.params(&params)) {
            lock.unlock();
            int rc;
            {
                std::lock_guard<std::mutex> turn(stream_lock(st));
                rc = launch_tiles((const void*)gpumpi_spread_params_kernel, &params, params.ntiles, st);
            }
            if (rc) return rc;
            CK(cudaStreamSynchronize(st));
            return GPUMPI_OK;
        }
    }
    // Build the used prefix on the host (zeros clear the flags), then copy it.
    unsigned char* img = g_noalloc_image;
    memset(img, 0, L.total);
    Job& job = *(Job*)(img + L.job);
    job.id = -2;
    job.timeout_ns = 30ull * 1000000000ull;
    job.status = (int*)(base + L.status);
    job.err_msg = base + L.err;
    CommShared& cs = *(CommShared*)(img + L.cs);
    cs.size = nranks;
    cs.ctx = 1;
    cs.members = nullptr;
    cs.pub = (Pub*)(base + L.pub);
    cs.arrive = (u64*)(base + L.flags);
    cs.mid = cs.arrive + nranks;
    cs.depart = cs.arrive + 2 * (size_t)nranks;
    MPI_Comm_impl* h = (MPI_Comm_impl*)(img + L.handles);
    for (int r = 0; r < nranks; r++) {
        h[r].kind = 1;
        h[r].ctx = 1;
        h[r].size = nranks;
        h[r].rank = r;
        h[r].refcnt = 1;
        h[r].cs = (CommShared*)(base + L.cs);
        h[r].seq = 0;
    }
    DevComm& dc = *(DevComm*)(img + L.dcomm);
    dc.handles = (MPI_Comm_impl*)(base + L.handles);
    dc.size = nranks;
    void** ptrs = (void**)(img + L.ptrs);
    for (int r = 0; r < nranks; r++) {
        ptrs[r] = sendbufs[r];
        ptrs[nranks + r] = recvbufs[r];
    }
    DevDesc& d = *(DevDesc*)(img + L.desc);
    d.op = GPUMPI_COLL_ALLREDUCE;
    d.dtype = dtype;
    d.redop = redop;
    d.root = 0;
    d.count = count;
    d.comm = 0;
    d.esize = es;
    d.algo = 0;
    d.sbufs = (void**)(base + L.ptrs);
    d.rbufs = (void**)(base + L.ptrs) + nranks;
    int* first = (int*)(img + L.first);
    first[0] = 0;
    first[1] = 1;
    CK(cudaMemcpyAsync(base, img, L.total, cudaMemcpyHostToDevice, st));
    PlanArgs args;
    args.job = (Job*)(base + L.job);
    args.descs = (const DevDesc*)(base + L.desc);
    args.comm_first = (const int*)(base + L.first);
    args.slot_comm = nullptr;
    args.slot_rank = nullptr;
    args.comms = (const DevComm*)(base + L.dcomm);
    args.ordered = 0;
    args.pad = 0;
    int rc = launch((const void*)gpumpi_plan_kernel, nranks, threads_per_rank, smem, &args, st);
    if (rc) return rc;
    CK(cudaStreamSynchronize(st));
    int status[16];
    CK(cudaMemcpy(status, base + L.status, sizeof(status), cudaMemcpyDeviceToHost));
    if (status[1] != 0) {
        char m[160];
        snprintf(m, sizeof(m), "gpumpi_allreduce_noalloc: device error %d on rank %d", status[1], status[2]);
        set_last_error(m);
        return GPUMPI_EJOB;
    }
    return GPUMPI_OK;
}
