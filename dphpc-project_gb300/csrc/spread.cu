// Kernel and tile lists of the spread form (spread.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "redop.cuh"
#include "spread.cuh"

namespace gm {

// Element types of a fold; sums and products of unsigned types use the signed
// type's code (the same bits).
enum FoldType : int { FT_I8, FT_U8, FT_I16, FT_U16, FT_I32, FT_U32, FT_I64, FT_U64, FT_F32, FT_F64, FT_NONE };

// ------------------------------------------------------------------ device

// Entry i of a table of addresses (constant while a launch runs), in global
// memory or among the kernel's parameters.
template <class P>
static __device__ __forceinline__ P ld_ptr(P const* t, u32 i) {
    return t[i];
}

template <class V>
static __device__ __forceinline__ V ld_unit(const char* p) {
    return __ldcg(reinterpret_cast<const V*>(p));
}

static __device__ __forceinline__ u32 smem_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }

// Asynchronous copy of B bytes to shared memory; 16-byte copies bypass L1.
template <int B>
static __device__ __forceinline__ void cp_async(u32 dst, const char* src) {
    if constexpr (B == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(B) : "memory");
}
static __device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
static __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <class V>
static __device__ __noinline__ void fan_tile(const SpreadCall& c, u32 tile) {
    constexpr int U = 8;
    const u32 pieces = (u32)((c.nu + c.per - 1) / c.per);
    const u32 piece = tile % pieces;
    const u32 rest = tile / pieces;
    const u32 q = rest % c.nsrc, r0 = rest / c.nsrc * c.group;
    const u32 r1 = min(r0 + c.group, c.ndst);
    const u64 o0 = (u64)piece * c.per;
    const u64 o1 = min(o0 + c.per, c.nu);
    const char* s = ld_ptr(c.src, q);
    const u64 row = (u64)q * c.nu * sizeof(V);
    for (u64 o = o0 + threadIdx.x; o < o1; o += U * SP_T) {
        V v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (o + u * SP_T < o1) v[u] = ld_unit<V>(s + (o + u * SP_T) * sizeof(V));
        for (u32 r = r0; r < r1; r++) {
            V* d = reinterpret_cast<V*>(ld_ptr(c.dst, r) + row) + o;
#pragma unroll
            for (int u = 0; u < U; u++)
                if (o + u * SP_T < o1) d[u * SP_T] = v[u];
        }
    }
}

// Where a thread of a copy tile stands in the sequence of all rows: item o of
// block q of row r, each block of nu items; next() is `step` items further.
struct CopyPos {
    u32 o, q, r;
    u32 d_o, d_q, d_r;
    __device__ __forceinline__ CopyPos(u32 nu, u32 nsrc, u64 k, u32 step) {
        const u64 blk = k / nu;
        o = (u32)(k - blk * nu);
        r = (u32)(blk / nsrc);
        q = (u32)(blk - (u64)r * nsrc);
        d_o = step % nu;
        d_q = step / nu % nsrc;
        d_r = step / nu / nsrc;
    }
    __device__ __forceinline__ void next(u32 nu, u32 nsrc) {
        o += d_o;
        q += d_q;
        r += d_r;
        if (o >= nu) {
            o -= nu;
            q++;
        }
        if (q >= nsrc) {
            q -= nsrc;
            r++;
        }
    }
};

template <class V>
static __device__ __noinline__ void copy_tile(const SpreadCall& c, u32 tile, char* ring) {
    const u64 total = (u64)c.ndst * c.nsrc * c.nu;
    const u64 k0 = (u64)tile * c.per + threadIdx.x;
    const u64 k1 = min((u64)tile * c.per + c.per, total);
    const u32 n = k0 < k1 ? (u32)((k1 - k0 + SP_T - 1) / SP_T) : 0;   // this thread's units
    const u32 nu = (u32)c.nu, nsrc = c.nsrc;
    const u64 rs = c.rs;
    const char* const* src = c.src;
    char* const* dst = c.dst;
    CopyPos to(nu, nsrc, k0, SP_T);
    if constexpr (sizeof(V) >= 4) {
        // through the thread's own part of the ring, as stream_tile does
        constexpr u32 GL = 4, NG = SP_RING / (SP_T * sizeof(V)) / GL;
        const u32 mine = smem_addr(ring) + threadIdx.x * (u32)sizeof(V);
        const V* slot = reinterpret_cast<const V*>(ring) + threadIdx.x;
        CopyPos from = to;
        u32 issued = 0, ig = 0, cg = 0;
        auto issue = [&]() {
#pragma unroll
            for (u32 g = 0; g < GL; g++) {
                if (issued < n) {
                    cp_async<sizeof(V)>(mine + (ig * GL + g) * (u32)(SP_T * sizeof(V)),
                                        ld_ptr(src, from.q) + rs * from.r + (u64)from.o * sizeof(V));
                    issued++;
                    from.next(nu, nsrc);
                }
            }
            cp_commit();
            if (++ig == NG) ig = 0;
        };
#pragma unroll 1
        for (u32 g = 0; g < NG - 1; g++) issue();
        for (u32 k = 0; k < n; k += GL) {
            issue();
            cp_wait<NG - 1>();
#pragma unroll
            for (u32 g = 0; g < GL; g++) {
                if (k + g < n) {
                    reinterpret_cast<V*>(ld_ptr(dst, to.r))[(u64)to.q * nu + to.o] = slot[(cg * GL + g) * SP_T];
                    to.next(nu, nsrc);
                }
            }
            if (++cg == NG) cg = 0;
        }
        cp_wait<0>();
    } else {
        for (u32 k = 0; k < n; k++) {
            reinterpret_cast<V*>(ld_ptr(dst, to.r))[(u64)to.q * nu + to.o] =
                ld_unit<V>(ld_ptr(src, to.q) + rs * to.r + (u64)to.o * sizeof(V));
            to.next(nu, nsrc);
        }
    }
}

// The same for blocks of a few hundred units and more: a warp takes SP_CHUNK units
// of a block at a time, four of a lane, which share the walk and the addresses.
// With a unit at a time those were most of the instructions: int32 Alltoall of the
// 16 communicators at 100003 per rank issued 0.63 instructions a clock and
// scheduler and reached 55 % of the DRAM rate; alone it takes 160 us so, 182 before.
template <class V>
static __device__ __noinline__ void chunk_tile(const SpreadCall& c, u32 tile, char* ring) {
    constexpr u32 GL = SP_CHUNK / 32, NG = SP_RING / (SP_T * sizeof(V)) / GL;
    const u32 nu = (u32)c.nu, nsrc = c.nsrc, lane = threadIdx.x & 31;
    const u32 len = (nu + SP_CHUNK - 1) / SP_CHUNK;   // chunks of a block
    const u64 total = (u64)c.ndst * nsrc * len;
    const u64 k0 = (u64)tile * c.per + (threadIdx.x >> 5);
    const u64 k1 = min((u64)tile * c.per + c.per, total);
    const u32 n = k0 < k1 ? (u32)((k1 - k0 + SP_WARPS - 1) / SP_WARPS) : 0;   // this warp's
    const u64 rs = c.rs;
    const char* const* src = c.src;
    char* const* dst = c.dst;
    const u32 mine = smem_addr(ring) + threadIdx.x * (u32)sizeof(V);
    const V* slot = reinterpret_cast<const V*>(ring) + threadIdx.x;
    CopyPos to(len, nsrc, k0, SP_WARPS), from = to;
    u32 issued = 0, ig = 0, cg = 0;
    auto issue = [&]() {
        if (issued < n) {
            const u32 at = from.o * SP_CHUNK + lane;
            const char* s = ld_ptr(src, from.q) + rs * from.r + (u64)at * sizeof(V);
#pragma unroll
            for (u32 g = 0; g < GL; g++)
                if (at + 32 * g < nu)
                    cp_async<sizeof(V)>(mine + (ig * GL + g) * (u32)(SP_T * sizeof(V)), s + 32 * g * sizeof(V));
            issued++;
            from.next(len, nsrc);
        }
        cp_commit();
        if (++ig == NG) ig = 0;
    };
#pragma unroll 1
    for (u32 g = 0; g < NG - 1; g++) issue();
    for (u32 k = 0; k < n; k++) {
        issue();
        cp_wait<NG - 1>();
        const u32 at = to.o * SP_CHUNK + lane;
        V* d = reinterpret_cast<V*>(ld_ptr(dst, to.r)) + (u64)to.q * nu + at;
#pragma unroll
        for (u32 g = 0; g < GL; g++)
            if (at + 32 * g < nu) d[32 * g] = slot[(cg * GL + g) * SP_T];
        to.next(len, nsrc);
        if (++cg == NG) cg = 0;
    }
    cp_wait<0>();
}

// Loads of a gather tile: the tile's n units of V of every source, one after
// another in g, SP_T units at a time.
template <class V>
static __device__ __forceinline__ void gather_load(const SpreadCall& c, u64 at, u32 n, char* g) {
    const u32 total = n * c.nsrc;
    const u32 d_q = SP_T / n, d_i = SP_T % n;
    u32 q = threadIdx.x / n, i = threadIdx.x % n;
    const u32 g_s = (u32)__cvta_generic_to_shared(g);
    for (u32 k = threadIdx.x; k < total; k += SP_T) {
        const char* p = ld_ptr(c.src, q) + at + (u64)i * sizeof(V);
        if constexpr (sizeof(V) >= 4) cp_async<sizeof(V)>(g_s + k * (u32)sizeof(V), p);
        else reinterpret_cast<V*>(g)[k] = ld_unit<V>(p);
        q += d_q;
        i += d_i;
        if (i >= n) {
            i -= n;
            q++;
        }
    }
}

// Stores of a gather tile: the n units of V at `res` to every destination.
template <class V>
static __device__ __forceinline__ void gather_store(const SpreadCall& c, u64 at, u32 n, const char* res) {
    const u32 total = n * c.ndst;
    const u32 d_r = SP_T / n, d_i = SP_T % n;
    u32 r = threadIdx.x / n, i = threadIdx.x % n;
    for (u32 k = threadIdx.x; k < total; k += SP_T) {
        reinterpret_cast<V*>(ld_ptr(c.dst, r) + at)[i] = reinterpret_cast<const V*>(res)[i];
        r += d_r;
        i += d_i;
        if (i >= n) {
            i -= n;
            r++;
        }
    }
}

template <class T, class O>
static __device__ __noinline__ void gather_tile(const SpreadCall& c, u32 tile, char* ring) {
    const u32 m = (u32)min((u64)c.per, c.nu - (u64)tile * c.per);
    const u64 at = c.off + tile * c.rs;
    if (c.ub == 16) gather_load<uint4>(c, at, m * (u32)sizeof(T) / 16, ring);
    else gather_load<T>(c, at, m, ring);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    const T* g = reinterpret_cast<const T*>(ring);
    // the results replace the first source's elements
    T* res = reinterpret_cast<T*>(ring);
    for (u32 i = threadIdx.x; i < m; i += SP_T) {
        T acc = g[i];
        u32 q = 1;
        for (; q + 8 <= c.nsrc; q += 8) {
            T x[8];
#pragma unroll
            for (int k = 0; k < 8; k++) x[k] = g[(q + k) * m + i];
#pragma unroll
            for (int k = 0; k < 8; k++) acc = O::f(x[k], acc);
        }
        for (; q < c.nsrc; q++) acc = O::f(g[q * m + i], acc);
        res[i] = acc;
    }
    __syncthreads();
    if (c.ub == 16) gather_store<uint4>(c, at, m * (u32)sizeof(T) / 16, ring);
    else gather_store<T>(c, at, m, ring);
}

// Where a call's addresses go in shared memory.
static __device__ __forceinline__ const char** src_table(char* smem) {
    return reinterpret_cast<const char**>(smem + SP_RING);
}
static __device__ __forceinline__ char** dst_table(char* smem) {
    return reinterpret_cast<char**>(smem + SP_RING) + SP_TAB;
}

// The call's addresses in shared memory (there already for a block's first
// tile), or where the host put them when they are many.  The block
// synchronises before it uses them.
static __device__ __forceinline__ void tables(const SpreadCall& c, char* smem, const char* const*& st,
                                              char* const*& dt) {
    st = c.src;
    dt = c.dst;
    const char** ts = src_table(smem);
    if (c.nsrc > SP_TAB || st == ts) return;
    char** td = dst_table(smem);
    for (u32 q = threadIdx.x; q < c.nsrc; q += SP_T) ts[q] = ld_ptr(c.src, q);
    for (u32 r = threadIdx.x; r < c.ndst; r += SP_T) td[r] = ld_ptr(c.dst, r);
    st = ts;
    dt = td;
}

// Every thread copies its own vectors into its own ring slots and reads only
// those, so the pipeline needs no barrier: cp.async groups complete in order
// and wait_group tells the thread when its oldest group has arrived.  GL loads
// make a group; the ring holds SP_RING bytes per block whatever the vector.
template <class T, class O, class V>
static __device__ __noinline__ void stream_tile(const SpreadCall& c, u32 tile, char* ring) {
    constexpr int B = sizeof(V);
    constexpr int GL = 4;
    constexpr int NG = (int)(SP_RING / (SP_T * B)) / GL;
    static_assert(NG >= 2, "ring");
    const char* const* st;
    char* const* dt;
    tables(c, ring, st, dt);
    __syncthreads();
    const u64 nvec = c.nu * sizeof(T) / B;
    const u64 v0 = (u64)tile * c.per * SP_T + threadIdx.x;
    const u32 rows = (u32)min((u64)c.per, (nvec - (u64)tile * c.per * SP_T + SP_T - 1) / SP_T);
    const u32 K = rows * c.nsrc;
    const u32 ng = (K + GL - 1) / GL;
    const u32 mine = (u32)__cvta_generic_to_shared(ring) + threadIdx.x * B;
    const V* slot = reinterpret_cast<const V*>(ring) + threadIdx.x;
    u64 iv = v0, cv = v0;
    u32 istep = 0, iq = 0, q = 0, ig = 0, cg = 0;
    auto issue = [&]() {
#pragma unroll
        for (int g = 0; g < GL; g++) {
            if (istep < K && iv < nvec) cp_async<B>(mine + (ig * GL + g) * (SP_T * B), st[iq] + c.off + iv * B);
            istep++;
            if (++iq == c.nsrc) {
                iq = 0;
                iv += SP_T;
            }
        }
        cp_commit();
        if (++ig == NG) ig = 0;
    };
#pragma unroll 1
    for (int g = 0; g < NG - 1; g++) issue();
    V acc{};
    for (u32 k = 0; k < ng; k++) {
        issue();   // into the slots that step k - 1 emptied
        cp_wait<NG - 1>();
#pragma unroll
        for (int g = 0; g < GL; g++) {
            if (k * GL + g < K) {
                const V x = slot[(cg * GL + g) * SP_T];
                if (q == 0) acc = x;
                else combine<T, O>(acc, x);
                if (++q == c.nsrc) {
                    if (cv < nvec)
                        for (u32 r = 0; r < c.ndst; r++) *reinterpret_cast<V*>(dt[r] + c.off + cv * B) = acc;
                    q = 0;
                    cv += SP_T;
                }
            }
        }
        if (++cg == NG) cg = 0;
    }
    cp_wait<0>();
}

// ---- SP_ROWS
//
// A warp folds chunks of `per` elements: it copies the 16-byte units that a
// chunk touches in `batch` sources at a time into its part of the ring, three
// such groups deep, and every lane folds every 32nd element from there.  So
// any element alignment costs the same: loads are 16-byte units, shared memory
// is read without bank conflicts and stores fill whole lines.  No bulk copies:
// one SM starts one of those every 44 cycles or so (measured with 144-byte
// rows), which 512-byte rows only just afford.
constexpr int SP_GROUPS = 3;

//
// MANY: more than SP_TAB ranks.  The sources' addresses are needed over and
// over, each before a load can start, and the shared memory that the blocks of
// an SM take leaves L1 no room for them: they lie at its end.  Of the
// destinations' addresses each lane reads one of 32 ahead of the stores before
// them, since a load from global memory cannot move above a store that may
// change it.  (Allreduce of 1024 ranks of 60001 FP64, chunks of 256 bytes, with
// all addresses in global memory 430 us, so 378; of 257 ranks 131 and 102.)
template <class T, class O, bool MANY>
static __device__ __noinline__ void rows_tile(const SpreadCall& c, u32 tile, char* smem) {
    constexpr int K = 16 / sizeof(T);    // elements a lane holds of a chunk of 512 bytes
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const char* const* st;
    char* const* dt;
    if constexpr (MANY) {
        const char** ts = reinterpret_cast<const char**>(smem + fold_table(c.nsrc));
        for (u32 q = threadIdx.x; q < c.nsrc; q += SP_T) ts[q] = ld_ptr(c.src, q);
        st = ts;
        dt = c.dst;
    } else {
        tables(c, smem, st, dt);
    }
    const u32 all = (u32)((c.nu + c.per - 1) / c.per);
    const u32 w0 = tile * c.rows + warp, w1 = min(tile * c.rows + c.rows, all);
    const u32 chunks = w1 > w0 ? (w1 - w0 + SP_WARPS - 1) / SP_WARPS : 0;   // this warp's
    const u32 groups = (c.nsrc + c.batch - 1) / c.batch;
    const u32 steps = chunks * groups;
    const u32 pitch = c.ub, units = pitch / 16, group_bytes = c.batch * pitch;
    char* part = smem + warp * (MANY ? rows_part(c.nsrc) : SP_PART);
    const u32 part_s = smem_addr(part);
    // unit `lane` of a group, and how units 32 further on lie
    const u32 j0 = lane / units, u0 = lane - j0 * units;
    const u32 d_j = 32 / units, d_u = 32 - d_j * units;
    u32 iw = w0, iq = 0, ig = 0, left = steps;
    auto issue = [&]() {
        if (left) {
            left--;
            const u64 e0 = (u64)iw * c.per;
            const u32 mb = (u32)min((u64)c.per, c.nu - e0) * (u32)sizeof(T);
            const u32 n = min(c.batch, c.nsrc - iq);
            const u64 at = c.off + e0 * sizeof(T);
            const u32 base = part_s + ig * group_bytes;
            u32 j = j0, u = u0;
            for (u32 k = lane; j < n; k += 32) {
                const uintptr_t a = (uintptr_t)st[iq + j] + at;
                if (u * 16 < ((u32)a & 15) + mb) cp_async<16>(base + k * 16, reinterpret_cast<const char*>((a & ~(uintptr_t)15) + u * 16));
                j += d_j;
                u += d_u;
                if (u >= units) {
                    u -= units;
                    j++;
                }
            }
            iq += c.batch;
            if (iq >= c.nsrc) {
                iq = 0;
                iw += SP_WARPS;
            }
        }
        cp_commit();
        if (++ig == SP_GROUPS) ig = 0;
    };
    __syncthreads();   // the tables
    for (int g = 0; g < SP_GROUPS - 1; g++) issue();
    u32 cg = 0;
    for (u32 w = w0; w < w1; w += SP_WARPS) {
        const u64 e0 = (u64)w * c.per;
        const u32 m = (u32)min((u64)c.per, c.nu - e0);
        const u64 at = c.off + e0 * sizeof(T);
        T acc[K];
        for (u32 q0 = 0; q0 < c.nsrc; q0 += c.batch) {
            __syncwarp();   // the group before has been read
            issue();
            cp_wait<SP_GROUPS - 1>();
            __syncwarp();   // every lane's part of this group is there
            const u32 n = min(c.batch, c.nsrc - q0);
            const char* row = part + cg * group_bytes + lane * (u32)sizeof(T);
            auto fold = [&](u32 j, bool first) {
                const T* r = reinterpret_cast<const T*>(row + j * pitch + (((u32)(uintptr_t)st[q0 + j] + (u32)at) & 15));
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (k * 32 < m) {   // the lanes past the chunk's end fold what is there, and store nothing
                        const T x = r[k * 32];
                        acc[k] = first ? x : O::f(x, acc[k]);
                    }
                }
            };
            u32 j = 0;
            if (q0 == 0) fold(j++, true);
#pragma unroll 4
            for (; j < n; j++) fold(j, false);
            if (++cg == SP_GROUPS) cg = 0;
        }
        if constexpr (MANY) {
            u64 next = lane < c.ndst ? (u64)ld_ptr(dt, lane) : 0;
            for (u32 r0 = 0; r0 < c.ndst; r0 += 32) {
                const u64 now = next;
                if (r0 + 32 + lane < c.ndst) next = (u64)ld_ptr(dt, r0 + 32 + lane);
                const u32 n = min(32u, c.ndst - r0);
#pragma unroll 4
                for (u32 r = 0; r < n; r++) {
                    T* d = reinterpret_cast<T*>(__shfl_sync(~0u, now, r) + at) + lane;
#pragma unroll
                    for (int k = 0; k < K; k++)
                        if (k * 32 + lane < m) d[k * 32] = acc[k];
                }
            }
        } else {
#pragma unroll 4
            for (u32 r = 0; r < c.ndst; r++) {
                T* d = reinterpret_cast<T*>(dt[r] + at) + lane;
#pragma unroll
                for (int k = 0; k < K; k++)
                    if (k * 32 + lane < m) d[k * 32] = acc[k];
            }
        }
    }
    cp_wait<0>();
}

// n units of V of each of nsrc sources, one after another in g, SP_T units at a time.
template <class V>
static __device__ __forceinline__ void passes_load(const char* const* src, u32 nsrc, u64 at, u32 n, char* g) {
    const u32 total = n * nsrc;
    const u32 d_q = SP_T / n, d_i = SP_T % n;
    u32 q = threadIdx.x / n, i = threadIdx.x % n;
    const u32 g_s = smem_addr(g);
    for (u32 k = threadIdx.x; k < total; k += SP_T) {
        const char* p = src[q] + at + (u64)i * sizeof(V);
        if constexpr (sizeof(V) >= 4) cp_async<sizeof(V)>(g_s + k * (u32)sizeof(V), p);
        else reinterpret_cast<V*>(g)[k] = ld_unit<V>(p);
        q += d_q;
        i += d_i;
        if (i >= n) {
            i -= n;
            q++;
        }
    }
}

// The n units of V at `res` to each of ndst destinations.
template <class V>
static __device__ __forceinline__ void passes_store(char* const* dst, u32 ndst, u64 at, u32 n, const char* res) {
    const u32 total = n * ndst;
    const u32 d_r = SP_T / n, d_i = SP_T % n;
    u32 r = threadIdx.x / n, i = threadIdx.x % n;
    for (u32 k = threadIdx.x; k < total; k += SP_T) {
        reinterpret_cast<V*>(dst[r] + at)[i] = reinterpret_cast<const V*>(res)[i];
        r += d_r;
        i += d_i;
        if (i >= n) {
            i -= n;
            r++;
        }
    }
}

// acc folded with n elements at g, `pitch` elements apart.
template <class T, class O>
static __device__ __forceinline__ T fold_column(T acc, const T* g, u32 n, u32 pitch) {
    u32 q = 0;
    for (; q + 8 <= n; q += 8) {
        T x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = g[(q + k) * pitch];
#pragma unroll
        for (int k = 0; k < 8; k++) acc = O::f(x[k], acc);
    }
    for (; q < n; q++) acc = O::f(g[q * pitch], acc);
    return acc;
}

// One chunk by the whole block (SP_ROWS with `group` 1): a gather tile in passes
// over the sources, each loaded into one half of the ring while the one before
// it is folded from the other.  More ranks than the ring holds 32 elements of
// would leave a gather tile with less than a warp's lanes to add, and an FP64
// addition takes a warp as long for one lane as for 32; a warp with a chunk of
// its own takes five times as long for each source, finding its address and
// its element there, and a call of few chunks has few warps.
template <class T, class O>
static __device__ __noinline__ void passes_tile(const SpreadCall& c, u32 tile, char* smem) {
    const u32 m = (u32)min((u64)c.per, c.nu - (u64)tile * c.per);
    const u64 at = c.off + (u64)tile * c.per * sizeof(T);
    const u32 batch = passes_half(c.nsrc) / (c.per * (u32)sizeof(T));   // sources of a pass
    const bool units16 = c.ub == c.per * sizeof(T);
    const char** ts = reinterpret_cast<const char**>(smem + fold_table(c.nsrc));
    for (u32 q = threadIdx.x; q < c.nsrc; q += SP_T) ts[q] = ld_ptr(c.src, q);
    __syncthreads();
    const u32 half = passes_half(c.nsrc);
    u32 q1 = 0, into = 0;   // the next pass to load and its half
    auto issue = [&]() {
        const u32 n = min(batch, c.nsrc - q1);
        if (n) {
            if (units16) passes_load<uint4>(ts + q1, n, at, m * (u32)sizeof(T) / 16, smem + into * half);
            else passes_load<T>(ts + q1, n, at, m, smem + into * half);
        }
        cp_commit();
        q1 += n;
        into ^= 1;
    };
    issue();
    T acc{};
    u32 from = 0;
    for (u32 q = 0; q < c.nsrc; q += batch) {
        issue();
        cp_wait<1>();
        __syncthreads();   // every thread's part of the pass has arrived
        const T* g = reinterpret_cast<const T*>(smem + from * half) + threadIdx.x;
        const u32 n = min(batch, c.nsrc - q);
        if (threadIdx.x < m) acc = q ? fold_column<T, O>(acc, g, n, m) : fold_column<T, O>(g[0], g + m, n - 1, m);
        from ^= 1;
        __syncthreads();   // before its half is loaded again
    }
    cp_wait<0>();
    // the results and the destinations' addresses take the ring's place
    char** td = reinterpret_cast<char**>(smem + SP_T * sizeof(T));
    if (threadIdx.x < m) reinterpret_cast<T*>(smem)[threadIdx.x] = acc;
    for (u32 r = threadIdx.x; r < c.ndst; r += SP_T) td[r] = ld_ptr(c.dst, r);
    __syncthreads();
    if (units16) passes_store<uint4>(td, c.ndst, at, m * (u32)sizeof(T) / 16, smem);
    else passes_store<T>(td, c.ndst, at, m, smem);
}

// The forms of more than SP_TAB ranks behind one call: with their choice on the way
// of every fold, ten short plain calls of 64 ranks took 63.7 us, so 62.6.
template <class T, class O>
static __device__ __noinline__ void many_tile(const SpreadCall& c, u32 tile, char* smem) {
    if (c.group) passes_tile<T, O>(c, tile, smem);
    else rows_tile<T, O, true>(c, tile, smem);
}

template <class T, class O>
static __device__ __forceinline__ void fold_tile(const SpreadCall& c, u32 tile, char* smem) {
    if (c.kind == SP_GATHER) gather_tile<T, O>(c, tile, smem);
    else if (c.kind == SP_STREAM) stream_tile<T, O, uint4>(c, tile, smem);
    else if (c.nsrc > SP_TAB) many_tile<T, O>(c, tile, smem);
    else rows_tile<T, O, false>(c, tile, smem);
}

// ---- bulk copies into the ring
//
// Every warp has its own part of the ring, cut into stages, and its own
// barriers: one lane loads a row into a stage by a bulk copy, the warp waits
// for it, uses it, and loads the stage again.  No block barrier is on the way.
struct Ring {
    u64 full[SP_WARPS][SP_MAX_STAGES];
    u32 failed;     // a wait ran out: the block's later waits return at once
};

static __device__ __forceinline__ u32 bar_done(u32 bar, u32 parity) {
    u32 done;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done;
}

// Wait for the loads of the warp's stage; bit `stage` of phases is the parity
// to wait for.  After the job's time limit the launch is marked failed.
static __device__ __forceinline__ void ring_wait(Ring& ring, u32 stage, u32& phases, Job* job) {
    const u32 bar = smem_addr(&ring.full[threadIdx.x >> 5][stage]);
    const u32 parity = (phases >> stage) & 1;
    phases ^= 1u << stage;
    if (bar_done(bar, parity)) return;
    const u64 t0 = gtime();
    while (!bar_done(bar, parity)) {
        if (*(volatile u32*)&ring.failed) return;
        if (gtime() - t0 > job->timeout_ns) {
            job_fail(job, (int)blockIdx.x, GPUMPI_ERR_TIMEOUT, "a bulk load did not complete");
            *(volatile u32*)&ring.failed = 1;
        }
    }
}

// Load `bytes` (a multiple of 16, may be 0) from src to dst for the warp's stage.
static __device__ __forceinline__ void ring_load(Ring& ring, u32 stage, char* dst, const char* src, u32 bytes) {
    const u32 bar = smem_addr(&ring.full[threadIdx.x >> 5][stage]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    if (bytes)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// ---- SP_MOVE

// A row in the ring.
struct MoveRow {
    u64 dst;           // address (one destination) or offset in every destination
    const char* src;   // first byte of the row
    u32 at, len;       // bytes in shared memory: the first one's place, how many
    u32 head, tail;    // bytes before and after them that were not loaded (a row at its buffer's start or end)
    u32 r0, pad;
};
static_assert(sizeof(MoveRow) * SP_WARPS * SP_MAX_STAGES <= 2 * SP_TAB * sizeof(char*), "row table");

// L2 policies of a copy's stores: FAN copies store far more than they read, and
// storing with evict_first leaves L2 to the few lines they read again (Bcast of
// the 16 communicators at 2^20 FP64 per rank 1329 -> 1250 us, at 2^15 56 -> 48 us;
// neither Alltoall nor Allreduce gain from it).  Launches that fit L2 keep their
// results there.
static __device__ __forceinline__ u64 l2_policy(bool cold) {
    u64 first, normal;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
    return cold ? first : normal;
}

// *p = v; FAN: under an L2 policy.
template <bool FAN, class V>
static __device__ __forceinline__ void st_move(V* p, const V& v, u64 policy) {
    if constexpr (!FAN) {
        *p = v;
    } else if constexpr (sizeof(V) == 16) {
        asm volatile("st.global.L2::cache_hint.v4.b32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
                     "r"(v.w), "l"(policy) : "memory");
    } else if constexpr (sizeof(V) == 8) {
        asm volatile("st.global.L2::cache_hint.v2.b32 [%0], {%1, %2}, %3;" ::"l"(p), "r"(v.x), "r"(v.y), "l"(policy)
                     : "memory");
    } else {
        asm volatile("st.global.L2::cache_hint.b32 [%0], %1, %2;" ::"l"(p), "r"(v), "l"(policy) : "memory");
    }
}

template <bool FAN, class V>
static __device__ __forceinline__ void move_units(char* d, const char* s, u32 n, u32 lane, u64 policy) {
    V* dv = reinterpret_cast<V*>(d);
    const V* sv = reinterpret_cast<const V*>(s);
    u32 i = lane;
    for (; i + 96 < n; i += 128) {
        const V a = sv[i], b = sv[i + 32], e = sv[i + 64], f = sv[i + 96];
        st_move<FAN>(dv + i, a, policy);
        st_move<FAN>(dv + i + 32, b, policy);
        st_move<FAN>(dv + i + 64, e, policy);
        st_move<FAN>(dv + i + 96, f, policy);
    }
    for (; i < n; i += 32) st_move<FAN>(dv + i, sv[i], policy);
}

// n bytes from shared memory s to d by one warp: the widest unit that both
// alignments share, bytes up to the first and after the last whole one; with
// no common alignment of 4, destination words put together from two source words.
template <bool FAN>
static __device__ __forceinline__ void move_row(char* d, const char* s, u32 n, u32 lane, u64 policy) {
    const u32 delta = ((u32)(uintptr_t)d - smem_addr(s)) & 15;
    const u32 unit = delta == 0 ? 16 : delta == 8 ? 8 : 4;
    u32 h = (0u - (u32)(uintptr_t)d) & (unit - 1);
    if (h > n) h = n;
    const u32 nw = (n - h) / unit;
    if (unit == 16) {
        move_units<FAN, uint4>(d + h, s + h, nw, lane, policy);
    } else if (unit == 8) {
        move_units<FAN, uint2>(d + h, s + h, nw, lane, policy);
    } else if ((delta & 3) == 0) {
        move_units<FAN, u32>(d + h, s + h, nw, lane, policy);
    } else {
        const u32* w = reinterpret_cast<const u32*>(reinterpret_cast<uintptr_t>(s + h) & ~(uintptr_t)3);
        const u32 sh = (smem_addr(s + h) & 3) * 8;
        for (u32 i = lane; i < nw; i += 32)
            st_move<FAN>(reinterpret_cast<u32*>(d + h) + i, __funnelshift_r(w[i], w[i + 1], sh), policy);
    }
    // at most 15 bytes on either side
    const u32 done = h + nw * unit;
    if (lane < h) d[lane] = s[lane];
    if (done + lane < n) d[done + lane] = s[done + lane];
}

template <bool FAN>
static __device__ __noinline__ void move_tile(const SpreadCall& c, u32 tile, char* smem, Ring& ring, u32& phases,
                                              Job* job) {
    const u64 policy = FAN ? l2_policy(c.cold) : 0;
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 pieces = (u32)((c.nu + c.per - 1) / c.per);
    const u32 sets = (c.ndst + c.group - 1) / c.group;   // of destinations
    const u32 all = pieces * c.nsrc * sets;
    const u32 row0 = tile * c.rows, row1 = min(row0 + c.rows, all);
    const u32 n = row1 - row0 > warp ? (row1 - row0 - warp + SP_WARPS - 1) / SP_WARPS : 0;   // this warp's rows
    const u32 pitch = c.per + 32;
    const u64 extent = c.rs ? c.rs * c.ndst : c.nu;   // bytes of a source buffer
    char* part = smem + warp * SP_PART;
    MoveRow* info = reinterpret_cast<MoveRow*>(smem + SP_RING) + warp * SP_MAX_STAGES;
    // lane i of 32 prepares rows i, 32 + i, ... of the warp and loads them when their turn comes
    MoveRow m;
    const char* from = nullptr;
    u32 bytes = 0;
    auto prepare = [&](u32 i) {
        if (i >= n) return;
        const u32 row = row0 + i * SP_WARPS + warp;
        // Alltoall: a destination's rows follow each other; else a piece's rows do,
        // which all read it while it is in L2
        u32 piece, q, r0;
        if (!FAN) {
            piece = row % pieces;
            q = row / pieces % c.nsrc;
            r0 = row / pieces / c.nsrc;
        } else {
            r0 = row % sets * c.group;
            piece = row / sets % pieces;
            q = row / sets / pieces;
        }
        const u64 p0 = (u64)piece * c.per;
        const u32 len = (u32)min((u64)c.per, c.nu - p0);
        const u64 off = c.rs * r0 + p0;
        m.src = ld_ptr(c.src, q) + off;
        m.dst = (u64)q * c.nu + p0;
        if (!FAN) m.dst += (u64)ld_ptr(c.dst, r0);
        // the 16-byte units the row touches, but none that leave the buffer
        const uintptr_t a = (uintptr_t)m.src, e = a + len;
        const uintptr_t x0 = off >= 16 ? a & ~(uintptr_t)15 : (a + 15) & ~(uintptr_t)15;
        const uintptr_t x1 = off + len + 16 <= extent ? (e + 15) & ~(uintptr_t)15 : e & ~(uintptr_t)15;
        from = reinterpret_cast<const char*>(x0);
        bytes = x1 > x0 ? (u32)(x1 - x0) : 0;
        m.head = bytes ? (x0 > a ? (u32)(x0 - a) : 0) : len;
        m.tail = bytes && e > x1 ? (u32)(e - x1) : 0;
        m.len = len - m.head - m.tail;
        m.at = x0 < a ? (u32)(a - x0) : 0;
        m.r0 = r0;
    };
    auto issue = [&](u32 i, u32 stage) {
        if ((i & 31) == 0) prepare(i + lane);
        if (lane == (i & 31)) {
            info[stage] = m;
            ring_load(ring, stage, part + stage * pitch, from, bytes);
        }
    };
    // the ring may hold what other tiles wrote with ordinary stores
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    for (u32 i = 0; i < c.stages && i < n; i++) issue(i, i);
    u32 stage = 0;
    for (u32 i = 0; i < n; i++) {
        ring_wait(ring, stage, phases, job);
        const MoveRow w = info[stage];
        const char* at = part + stage * pitch + w.at;
        const u32 r1 = FAN ? min(w.r0 + c.group, c.ndst) : w.r0 + 1;
        // rows whose 16-byte units are also their destinations' leave by bulk
        // copies, a lane for each destination; the rest go through registers
        const bool whole = ((w.at | w.len | w.head | w.tail) & 15) == 0 && w.head + w.tail == 0;
        for (u32 rb = w.r0; rb < r1; rb += 32) {
            const u32 r = rb + lane;
            const u64 d = r < r1 ? (FAN ? (u64)ld_ptr(c.dst, r) + w.dst : w.dst) : 0;
            const bool bulk = whole && (d & 15) == 0;
            if (FAN && bulk && r < r1)
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;"
                             ::"l"(d), "r"(smem_addr(at)), "r"(w.len), "l"(policy) : "memory");
            else if (bulk && r < r1)
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                             ::"l"(d), "r"(smem_addr(at)), "r"(w.len) : "memory");
            u32 rest = __ballot_sync(~0u, r < r1 && !bulk);
            while (rest) {
                const u32 k = __ffs(rest) - 1;
                rest &= rest - 1;
                char* to = reinterpret_cast<char*>(__shfl_sync(~0u, d, k));
                move_row<FAN>(to + w.head, at, w.len, lane, policy);
                if (w.head | w.tail) {
                    for (u32 x = lane; x < w.head; x += 32) to[x] = __ldcg(w.src + x);
                    const u32 done = w.head + w.len;
                    for (u32 x = lane; x < w.tail; x += 32) to[done + x] = __ldcg(w.src + done + x);
                }
            }
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();   // the stage has been read
        if (i + c.stages < n && !*(volatile u32*)&ring.failed) issue(i + c.stages, stage);
        if (++stage == c.stages) stage = 0;
    }
    // the results are in global memory before the launch ends
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

template <template <class> class O>
static __device__ void fold_types(const SpreadCall& c, u32 tile, char* smem) {
    switch (c.fn >> 2) {
        case FT_I8: fold_tile<signed char, O<signed char>>(c, tile, smem); break;
        case FT_I16: fold_tile<short, O<short>>(c, tile, smem); break;
        case FT_I32: fold_tile<int, O<int>>(c, tile, smem); break;
        case FT_I64: fold_tile<long long, O<long long>>(c, tile, smem); break;
        case FT_F32: fold_tile<float, O<float>>(c, tile, smem); break;
        case FT_F64: fold_tile<double, O<double>>(c, tile, smem); break;
        default: break;
    }
}

template <template <class> class O>
static __device__ void fold_unsigned(const SpreadCall& c, u32 tile, char* smem) {
    switch (c.fn >> 2) {
        case FT_U8: fold_tile<unsigned char, O<unsigned char>>(c, tile, smem); break;
        case FT_U16: fold_tile<unsigned short, O<unsigned short>>(c, tile, smem); break;
        case FT_U32: fold_tile<unsigned, O<unsigned>>(c, tile, smem); break;
        case FT_U64: fold_tile<unsigned long long, O<unsigned long long>>(c, tile, smem); break;
        default: break;
    }
}

static __device__ void run_tile(const SpreadCall& c, u32 tile, char* smem, Ring& ring, u32& phases, Job* job) {
    if (c.kind == SP_MOVE) {
        if (c.rs) move_tile<false>(c, tile, smem, ring, phases, job);
        else move_tile<true>(c, tile, smem, ring, phases, job);
    } else if (c.kind == SP_FAN) {
        switch (c.ub) {
            case 16: fan_tile<uint4>(c, tile); break;
            case 8: fan_tile<uint2>(c, tile); break;
            case 4: fan_tile<u32>(c, tile); break;
            case 2: fan_tile<unsigned short>(c, tile); break;
            default: fan_tile<unsigned char>(c, tile); break;
        }
    } else if (c.kind == SP_COPY) {
        switch (c.group ? c.ub + 1 : c.ub) {
            case 9: chunk_tile<uint2>(c, tile, smem); break;
            case 5: chunk_tile<u32>(c, tile, smem); break;
            case 16: copy_tile<uint4>(c, tile, smem); break;
            case 8: copy_tile<uint2>(c, tile, smem); break;
            case 4: copy_tile<u32>(c, tile, smem); break;
            case 2: copy_tile<unsigned short>(c, tile, smem); break;
            default: copy_tile<unsigned char>(c, tile, smem); break;
        }
    } else {
        switch (c.fn & 3) {
            case GPUMPI_OP_MAX:
                fold_types<OMax>(c, tile, smem);
                fold_unsigned<OMax>(c, tile, smem);
                break;
            case GPUMPI_OP_MIN:
                fold_types<OMin>(c, tile, smem);
                fold_unsigned<OMin>(c, tile, smem);
                break;
            case GPUMPI_OP_SUM: fold_types<OSum>(c, tile, smem); break;
            default: fold_types<OProd>(c, tile, smem); break;
        }
    }
}

// Shared state of a block: its current call and the ring's barriers.
struct Block {
    SpreadCall c;   // in shared memory, so that no thread holds it in registers
    u32 found;
    Ring ring;
};

// Launches of one stream overlap: the next one starts its blocks and reads its
// plan's tables while this one runs, and touches no buffer before grid_wait():
// everything the stream ran before it is then complete and visible.  A launch
// lets the next one start once it may run itself, so that no third launch waits
// in the SMs: with three, blocks went wherever one had just ended, several to
// one SM (Allreduce of 200 ranks of 50000 FP64 134 us, two launches 78 us).
// Back to back, an Allreduce of one FP64 value over 16 ranks takes 2.6 us instead
// of 5.1; alone, with a wait after each, 12.8 us either way.
static __device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
static __device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

static __device__ __forceinline__ void block_begin(Block& b) {
    if (threadIdx.x < SP_WARPS * SP_MAX_STAGES) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&b.ring.full[0][0] + threadIdx.x))
                     : "memory");
        b.ring.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

static __device__ __forceinline__ void block_end(Block& b) {
    if (b.ring.failed) {
        // loads may still be on their way into this block's shared memory
        const u64 t0 = gtime();
        while (gtime() - t0 < 1000000000ull) __nanosleep(1000);
    }
}

// The call whose range holds tile t, into b.c.  The block synchronises before
// it uses it.
static __device__ __forceinline__ void find_call(Block& b, const SpreadCall* one, const SpreadCall* calls, u32 ncalls,
                                                 u32 t) {
    constexpr u32 W = sizeof(SpreadCall) / 8;
    if (one) {
        if (threadIdx.x < W)
            reinterpret_cast<u64*>(&b.c)[threadIdx.x] = reinterpret_cast<const u64*>(one)[threadIdx.x];
        return;
    }
    for (u32 i = threadIdx.x; i < ncalls; i += SP_T) {   // exactly one thread finds it
        const u32 f = calls[i].first_tile, n = calls[i].ntiles;
        if (t - f < n) b.found = i;
    }
    __syncthreads();
    if (threadIdx.x < W)
        reinterpret_cast<u64*>(&b.c)[threadIdx.x] = reinterpret_cast<const u64*>(calls + b.found)[threadIdx.x];
}

// In the parameter form src and dst are indexes into ptrs.
static __device__ __forceinline__ void set_tables(Block& b, void* const* ptrs) {
    __syncthreads();
    if (!ptrs) return;
    if (threadIdx.x == 0) {
        b.c.src = reinterpret_cast<const char* const*>(ptrs + reinterpret_cast<size_t>(b.c.src));
        b.c.dst = reinterpret_cast<char* const*>(ptrs + reinterpret_cast<size_t>(b.c.dst));
    }
    __syncthreads();
}

// The call of this block's first tile and its addresses.  They are the plan's
// own and do not change, so this runs before the block waits for the launches
// ahead of it: three dependent loads from L2 that the tile no longer waits for
// (16 communicators of 4..256 ranks, 301 elements each, 18.8 -> 17.1 us).
static __device__ __forceinline__ void first_call(Block& b, const SpreadCall* one, const SpreadCall* calls, u32 ncalls,
                                                  u32 ntiles, char* smem, void* const* ptrs = nullptr) {
    if (blockIdx.x >= ntiles) return;
    find_call(b, one, calls, ncalls, blockIdx.x);
    set_tables(b, ptrs);
    // SP_MOVE keeps its rows where the tables would lie
    if (b.c.kind == SP_MOVE || b.c.nsrc > SP_TAB || b.c.ndst > SP_TAB) return;
    const char** ts = src_table(smem);
    char** td = dst_table(smem);
    for (u32 q = threadIdx.x; q < b.c.nsrc; q += SP_T) ts[q] = ld_ptr(b.c.src, q);
    for (u32 r = threadIdx.x; r < b.c.ndst; r += SP_T) td[r] = ld_ptr(b.c.dst, r);
    __syncthreads();
    if (threadIdx.x == 0) {
        b.c.src = ts;
        b.c.dst = td;
    }
}

// This block's tiles of a level, after first_call().
static __device__ __forceinline__ void run_tiles(Block& b, const SpreadCall* one, const SpreadCall* calls, u32 ncalls,
                                                 u32 ntiles, char* smem, u32& phases, Job* job,
                                                 void* const* ptrs = nullptr) {
    for (u32 t = blockIdx.x; t < ntiles; t += gridDim.x) {
        if (t != blockIdx.x) {
            find_call(b, one, calls, ncalls, t);
            set_tables(b, ptrs);
        } else {
            __syncthreads();
        }
        run_tile(b.c, t - b.c.first_tile, smem, b.ring, phases, job);
        __syncthreads();
    }
}

}  // namespace gm

using namespace gm;

extern "C" __global__ void __launch_bounds__(SP_T, SP_BLOCKS_PER_SM)
    gpumpi_spread_kernel(const __grid_constant__ SpreadArgs A) {
    extern __shared__ __align__(16) char sp_smem[];
    __shared__ Block b;
    u32 phases = 0;
    block_begin(b);
    const SpreadCall* one = A.ncalls == 1 ? &A.one : nullptr;
    first_call(b, one, A.calls, A.ncalls, A.ntiles, sp_smem);
    if (A.overlap) {
        if (threadIdx.x == 0) __threadfence();   // no line that L1 kept from before the first of them
    } else {
        grid_wait();   // blocks without a tile too: no launch ends before the ones it follows
    }
    grid_trigger();
    run_tiles(b, one, A.calls, A.ncalls, A.ntiles, sp_smem, phases, A.job);
    if (A.overlap && blockIdx.x == 0) grid_wait();   // no launch ends before the ones it follows
    block_end(b);
}

// One call whose descriptors and addresses come with the launch, for callers
// without device memory for them.
extern "C" __global__ void __launch_bounds__(SP_T, SP_BLOCKS_PER_SM)
    gpumpi_spread_params_kernel(const __grid_constant__ SpreadParams A) {
    extern __shared__ __align__(16) char sp_smem[];
    __shared__ Block b;
    u32 phases = 0;
    block_begin(b);
    first_call(b, nullptr, A.calls, A.ncalls, A.ntiles, sp_smem, A.ptrs);
    grid_wait();
    grid_trigger();
    run_tiles(b, nullptr, A.calls, A.ncalls, A.ntiles, sp_smem, phases, nullptr, A.ptrs);
    block_end(b);
}

// ------------------------------------------------------------------ host

namespace gm {

static int fold_type(int dtype) {
    switch (dtype) {
        case MPI_SIGNED_CHAR: case MPI_INT8_T: return FT_I8;
        case MPI_UNSIGNED_CHAR: case MPI_UINT8_T: case MPI_BYTE: return FT_U8;
        case MPI_SHORT: case MPI_INT16_T: return FT_I16;
        case MPI_UNSIGNED_SHORT: case MPI_UINT16_T: return FT_U16;
        case MPI_INT: case MPI_INT32_T: return FT_I32;
        case MPI_UNSIGNED: case MPI_UINT32_T: return FT_U32;
        case MPI_LONG: case MPI_LONG_LONG_INT: case MPI_LONG_LONG: case MPI_INT64_T: return FT_I64;
        case MPI_UNSIGNED_LONG: case MPI_UNSIGNED_LONG_LONG: case MPI_UINT64_T: return FT_U64;
        case MPI_FLOAT: return FT_F32;
        case MPI_DOUBLE: return FT_F64;
        default: return FT_NONE;
    }
}

// Alltoall blocks from here on move by bulk copies; shorter ones go one unit per
// thread (SP_COPY).  A row costs its warp some 80 instructions whatever its
// length, a unit per thread some 15 each, so with units of 4 bytes and more the
// lines cross near 8 KiB (16-byte units, int32 Alltoall of communicators of 4..256
// ranks, 2^17 elements per rank: 251 us with bulk copies from 2 KiB, 218 us from 8
// KiB; FP64 at 2^20 3.74 ms without them, 2.9 ms with.  4- and 8-byte units, the
// 16-communicator batch, from 512 bytes / 8 KiB: 2^14 per rank 195 / 180 us, 2^15
// 330 / 318, 30001 370 / 362; no difference to 16 and 32 KiB).  Units of 1 and 2
// bytes cannot take the ring and do so from 512 bytes.
constexpr u64 SP_MOVE_UNITS = 8192;
constexpr u64 SP_MOVE_BYTES = 512;
// Units of 1 byte of many ranks sooner: their rows fill every warp, and cost as much
// as some 250 units (odd uint8 Alltoall, SP_COPY / SP_MOVE, us: 64 ranks, blocks of 385
// bytes 6.3 / 6.8, 501 7.4 / 7.1; 256 ranks, 193 34 / 42, 257 44 / 43, 501 84 / 50; 1000
// ranks, 65 266 / 526, 129 387 / 404, 257 820 / 427, 501 1641 / 470, rank blocks 885).
static u64 move_bytes(u32 unit, u64 blocks) {
    return unit > 1 || blocks < 65536 ? SP_MOVE_BYTES : blocks < 524288 ? 257 : 144;
}
constexpr u64 SP_PIECE = 1920;       // longest piece: three fit a warp's part of the ring

// Bytes of a rank's vector from which a fold goes by rows instead of gather
// tiles.  A gather tile's loads are all under way at once, which the fewer
// warps of a small launch need; rows keep loads under way while they fold and
// take any alignment in 16-byte units, which counts in large launches.
// For calls among others, and lone ones above SP_LONE_BYTES.  Measured one call at
// a time with the tiles of such a level, gather -> rows, us: Allreduce FP64 of 64
// ranks, 50000 19.5 -> 27.7, 131072 57.9 -> 50.0, 400000 136 -> 98; 50001 23.0 ->
// 28.2, 131073 68 -> 50; of
// 200 ranks, 50000 62 -> 78, 131072 144 -> 140; int32 of 64 ranks, 50001 16.7 ->
// 15.3, 131073 33 -> 26; of the 16 communicators of 4..256 ranks, 2^15 FP64 151 ->
// 161, 2^16 234 -> 199, 2^16 int32 113 -> 115, 32769 int32 97 -> 89.
static u64 rows_min(bool aligned, double total) {
    const bool large = total >= 268435456.0;
    if (!aligned) return large ? 131072 : 524288;
    return large ? 524288 : 1048576;
}

// Bcast and Allgather by bulk copies: one load of a piece, a store to each of a
// group of destinations.  With 16-byte alignment the stores are bulk copies, one
// lane each, and the larger the group the better (2^20 FP64 per rank, group 8
// 1461 us, 32 1413 us, all 1336 us; pieces of 6272 bytes 1325 us); otherwise the
// warp writes one destination after another and 8 keep enough warps busy (100003
// int32: 8 74 us, 16 79 us, 32 103 us).  It takes a large launch to keep the
// pipelines full; before that, through registers (SP_FAN): Bcast of FP64 to 200
// ranks, 105 MB 21.4 us against 21.9, 210 MB 46.3 against 39.6; to 48 ranks, 50 MB
// 18.6 against 19.1, 400 MB 83 against 70; odd buffers, 210 MB 21.5 against 36.7
// and 420 MB 87.5 against 76.5; the 16-communicator batch at 500001 per rank 5364
// against 5104, at 50001 561 against 565.  (Lone calls up to SP_LONE_BYTES have
// their own rule in add().)
constexpr u64 SP_FAN_PIECE = 6272, SP_HALF_PIECE = 3072;
constexpr double SP_FAN_ALIGNED = 1024, SP_FAN_ODD = 8;
static u64 fan_min(bool units16, double total) {
    if (units16) return total >= 2e8 ? 8192 : ~0ull;
    return total >= 1e9 ? 524288 : ~0ull;
}

// A call that has a level to itself and moves up to this much is cut into one,
// two or four equal tiles for each SM, which all run at once: no tail, and no
// more of the 1 to 2 us with which a tile starts (its call, its addresses, the
// first loads) than it takes to keep loads under way.  Three tiles for each
// block that fits, as in a level of many calls, leave a tail and are short.
// Measured with 152, 304, 608 and 1216 tiles for each kind, 4..200 ranks, 0.1 to
// 200 MB, three tiles / these, us: Allreduce of 64 ranks of 15616 FP64 10.4 -> 6.4,
// of 124992 float32 16.6 -> 12.4; of 200 of 4992 FP64 32 -> 12.5; Reduce of 16 of
// 124992 float32 6.3 -> 3.6; Alltoall of 4 of 1 MB blocks 24.3 -> 8.6, of 64 of
// 7.8 KB 14.2 -> 8.6; Bcast of 32 MB to 64 ranks 10.5 -> 7.1.  The same for 200 MB
// (Alltoall 50 -> 36) but not much beyond.
constexpr double SP_LONE_BYTES = 2.5e8;
constexpr u32 SP_SMS = 152;

static u64 split(u64 units, u64 tiles) { return (units + tiles - 1) / tiles; }
static u64 round_up(u64 v, u64 step) { return (v + step - 1) / step * step; }

// Elements of a lone fold's gather tile, or 0 when the ring is too small for
// four tiles for each SM or a thread would fold more than two elements.  One
// tile for each SM is enough while a thread folds one (64 ranks of 3904 FP64: one
// 5.1, two 5.2, four 5.4 us; 4 of 62496: 3.3, 3.0, 3.1; 4 of 500000 float32, four
// tiles 5.3, SP_STREAM 4.6).
static u64 lone_gather(u64 n, u64 step, u64 fits) {
    for (u64 k = 1; k <= 4; k *= 2) {
        const u64 m = round_up(split(n, SP_SMS * k), step);
        if (m <= fits && m <= (k > 1 ? 2 : 1) * SP_T) return m;
    }
    return 0;
}

// Elements from which the rest of a fold of 1- or 2-byte elements goes on its own
// (Reduce of uint8 of odd lengths, rank blocks / single elements / so, us: 3 ranks of
// 3001, four calls 55 / 10.3 / 3.5; 64 of 600001 66 / 57 / 12; 256 of 40001 96 / 29 / 5.3,
// of 600001 651 / 382 / 41).
constexpr u64 GATHER_REST = 1024;
constexpr u64 RAGGED_BYTES = 4096;   // the same for the end of a Bcast

static bool is_fold(int op) { return op == GPUMPI_COLL_REDUCE || op == GPUMPI_COLL_ALLREDUCE; }

bool SpreadBuilder::covers(const gpumpi_coll_desc& d, int P, int esize) {
    if (d.op == GPUMPI_COLL_BARRIER || !d.recvbufs || P > SP_MAX_RANKS) return false;
    if ((d.algo != 0 && d.algo != tiles_schedule(d.op)) || d.sync != 0) return false;
    if (is_fold(d.op) && fold_type(d.dtype) == FT_NONE) return false;
    auto usable = [&](const void* p) { return p != nullptr && p != MPI_IN_PLACE && (uintptr_t)p % esize == 0; };
    for (int r = 0; r < P; r++) {
        if (d.op != GPUMPI_COLL_BCAST && !usable(d.sendbufs ? d.sendbufs[r] : d.recvbufs[r])) return false;
        if ((d.op != GPUMPI_COLL_REDUCE || r == d.root) && !usable(d.recvbufs[r])) return false;
    }
    return true;
}

void SpreadLoad::count(const gpumpi_coll_desc& d, int P, int esize) {
    const double e = (double)d.count * esize;
    calls++;
    switch (d.op) {
        case GPUMPI_COLL_BCAST: bytes += e * P; break;
        case GPUMPI_COLL_REDUCE: bytes += e * (P + 1); break;
        case GPUMPI_COLL_ALLREDUCE: bytes += 2 * e * P; break;
        default: bytes += 2 * e * P * P;
    }
    if (is_fold(d.op)) folded += (double)d.count;
}

void SpreadBuilder::add(const gpumpi_coll_desc& d, int P, int esize, const SpreadLoad& level) {
    if (d.count == 0) return;
    // Traffic of one tile in a level of several calls: 1.75 tiles for each of the
    // blocks that run at once in a short launch, three in a long one and for a
    // single large call (Allreduce of 8 ranks, 268 MB: 1.75 48.0, three 46.0 us).  More of them
    // even out the end, fewer start less often, each with its pipeline empty (the
    // 16-communicator batch with 1.25 / 1.75 / 2 / 3 of them, us: 700 per rank 17.4,
    // 17.5, 20.0, 20.9; 1500 30.1, 28.7, 29.7, 32.3; 4096 60.4, 57.7, 58.0, 62.2; 8192
    // 117, 103.5, 97.4, 102.0; 16384 218, 178.5, 178.4, 181.4; 24000 367, 297, 272, 261;
    // 32768 with 2 / 3 / 4 362, 319, 345).  At most 2 MB: 2^20 with 0.5 MiB 10.18 ms, 1
    // MiB 9.90, 2 MB 9.79, 8 MB 9.92.
    const double total = level.bytes;
    const bool alone = level.calls == 1, lone = alone && total <= SP_LONE_BYTES, large = alone && !lone;
    const double waves = level.calls == 1 || total >= 1.1e9 ? 3 : total < 3.2e8 ? 1.75 : 2;
    const double target = lone ? total / (SP_SMS * 2)
                               : std::min(2e6, std::max(16384.0, total / (SP_SMS * SP_BLOCKS_PER_SM * waves)));
    std::vector<void*> src, dst;
    auto sendbuf = [&](int r) { return d.sendbufs ? d.sendbufs[r] : d.recvbufs[r]; };
    switch (d.op) {
        case GPUMPI_COLL_BCAST:
            src.push_back(d.recvbufs[d.root]);
            for (int r = 0; r < P; r++)
                if (r != d.root && d.recvbufs[r] != d.recvbufs[d.root]) dst.push_back(d.recvbufs[r]);
            break;
        case GPUMPI_COLL_REDUCE:
            for (int r = 0; r < P; r++) src.push_back(sendbuf(r));
            dst.push_back(d.recvbufs[d.root]);
            break;
        default:
            for (int r = 0; r < P; r++) {
                src.push_back(sendbuf(r));
                dst.push_back(d.recvbufs[r]);
            }
    }
    if (dst.empty() || (P == 1 && src[0] == dst[0])) return;
    uintptr_t bits = 0;   // alignment that every address shares
    for (void* p : src) bits |= (uintptr_t)p;
    for (void* p : dst) bits |= (uintptr_t)p;
    SpreadCall c;
    memset(&c, 0, sizeof(c));
    c.src = (const char* const*)ptrs.size();
    ptrs.insert(ptrs.end(), src.begin(), src.end());
    c.dst = (char* const*)ptrs.size();
    ptrs.insert(ptrs.end(), dst.begin(), dst.end());
    c.nsrc = (u32)src.size();
    c.ndst = (u32)dst.size();
    u64 bytes = d.count * (u64)esize;
    if (is_fold(d.op)) {
        int ft = fold_type(d.dtype);
        if (d.redop == GPUMPI_OP_SUM || d.redop == GPUMPI_OP_PROD) {
            if (ft == FT_U8 || ft == FT_U16 || ft == FT_U32 || ft == FT_U64) ft--;
        }
        c.fn = ft * 4 + d.redop;
        const u64 V = 16 / esize, n = d.count;
        const bool aligned = bits % 16 == 0;
        const double row = (double)(c.nsrc + c.ndst);   // traffic per byte of a row
        auto gather = [&](u64 first, u64 count, u64 per, u64 distance) {
            SpreadCall g = c;
            g.kind = SP_GATHER;
            g.off = first * esize;
            g.nu = count;
            g.per = (u32)per;
            g.rs = distance * esize;
            g.ub = aligned && count % V == 0 && per % V == 0 && distance % V == 0 ? 16 : esize;
            g.ntiles = (u32)((count + per - 1) / per);
            g.tile_bytes = (u32)(row * per * esize);
            calls.push_back(g);
        };
        // whole vectors, or what lies 16 bytes and more from both ends of the buffers
        const u64 lo = aligned ? 0 : V, hi = aligned ? n / V * V : n > 2 * V ? n - V : 0;
        // 1- and 2-byte types take gather tiles of whole vectors and one of the rest: loaded
        // one by one their elements are most of a tile's work
        const bool rest = aligned && esize < 4 && n % V && n >= GATHER_REST;
        const u64 step = aligned && (rest || n % V == 0) ? V : 1;
        auto gather_all = [&](u64 per) {
            gather(0, rest ? hi : n, per, per);
            if (rest) gather(hi, n - hi, n - hi, n - hi);
        };
        const double fits = (double)SP_RING / ((double)P * esize);
        const u64 most = (u64)fits / step * step;   // elements of the largest gather tile
        const u64 nrows = split(hi / V, SP_T);
        // Above SP_TAB ranks gather tiles stay where they all run at once, which is
        // short calls; then SP_ROWS in passes, with as few elements a tile as keep the SMs
        // busy (512 bytes at most); from 576 KiB chunks of a warp, whose loads never pause
        // (1- and 2-byte types from 1 MiB, from 96 KiB in odd buffers, which passes load one by one;
        // Reduce of FP64, passes / chunks: 512 ranks of 63476 95 / 124, of 97656 138 / 127
        // us, 320 of 50780 75 / 102, of 101560 93 / 83).
        // One call, Reduce of FP64 unless named, gather / passes of 32, 64, 128 elements
        // / a warp's chunks of 512 bytes, us: 1024 ranks of 2000 48 / 51, 58, 73 / 240,
        // of 20000 298 / 107, 86, 107 / 254, of 60000 835 / 216, 174, 166 / 257, of
        // 150000 1897 / 443, 344, 324 / 312; 512 of 60000 256 / 115, 92, 86 / 131, of
        // 150000 525 / 237, 181, 168 / 158; Allreduce of 60001 int32, 1024 ranks 279 /
        // 156, 147, 142 / 175, of 150001 448 / 354, 320, 292 / 277; of 512 ranks of
        // 150001 uint8 320 / -, -, 244 / 206.
        // (Rank blocks: Reduce of 60000, 512 ranks 145, 1024 277.)  Among other calls
        // the warps' chunks start earlier (Allreduce and Reduce of FP64 and int32 by
        // communicators of 1024, 512, 256 and 64 ranks, passes / chunks from 128 KiB:
        // 20001 elements 384 / 559, 60001 1010 / 801).
        const bool many = P > SP_TAB;
        if (lone) {
            const u64 m = lone_gather(n, step, most);
            if (m) {
                gather_all(m);
                return;
            }
        }
        // A lone fold that does not fit streams when that gives two tiles for each
        // SM (4 ranks of 10^6 FP64: rows 13.7, stream 12.3, gather 14.6 us; 64 of
        // 62496, 122 rows: 23.0, 19.3, 18.7; 200 of 20000, 39 rows: 52, 52, 26)
        if (aligned && !many && (lone ? nrows >= 2 * SP_SMS : row * SP_T * 16 <= 2 * target) && hi >= SP_T * V) {
            c.kind = SP_STREAM;
            c.nu = hi;
            c.per = (u32)std::max(1.0, std::min((double)nrows, target / (row * SP_T * 16)));
            if (lone) c.per = (u32)split(nrows, 2 * SP_SMS);
            c.ntiles = (u32)((nrows + c.per - 1) / c.per);
            c.tile_bytes = (u32)(row * SP_T * 16 * c.per);
            calls.push_back(c);
            if (hi < n) gather(hi, n - hi, n - hi, n - hi);
            return;
        }
        // a lone fold of buffers aligned to their elements (4 ranks of 2 * 10^6 int32:
        // gather 19.4, rows 13.7 us; 64 of 62497 FP64, 500 KB each: 20.0, 24.6 us)
        const u64 inner = hi > lo ? (hi - lo) * esize : 0;
        // From 250 MB a single call always goes by rows: even of 256 ranks it has 1000
        // chunks, a gather tile of many ranks a few elements (Reduce of 256 ranks of
        // 1015624 uint8: gather 682, rows 93 us; Allreduce of 160 of 812500 446, 96).
        const u64 least = many && alone ? esize >= 4 ? 589824 : aligned ? 1048576 : 98304
                          : large      ? 0
                          : lone        ? aligned ? ~0ull : 524288
                          : many        ? std::max<u64>(32768 * esize, rows_min(aligned, total))
                                        : rows_min(aligned, total);
        const bool passes = many && inner && inner < least && (aligned || esize > 1) &&
                            (lone || (level.folded > 4.0 * SP_SMS * most && (alone || n > SP_SMS / 2 * most)));
        if (passes || (inner && inner >= least)) {
            c.kind = SP_ROWS;
            c.off = lo * esize;
            c.nu = hi - lo;
            u32 chunk = 512;
            if (passes) {
                const u32 per = level.folded <= 2.0 * SP_SMS * 32    ? 32
                                : level.folded <= 4.0 * SP_SMS * 64  ? 64
                                : level.folded <= 4.0 * SP_SMS * 128 ? 128
                                                                     : 256;
                chunk = std::min(512u, per * (u32)esize);
                c.group = 1;
            }
            while (many && alone && !passes && chunk > 128 && inner < 580ull * chunk) chunk /= 2;
            while (!(many && alone) && !large && !passes && chunk > 32 * (u32)esize && row * chunk * SP_WARPS > 4 * target) chunk /= 2;
            c.per = chunk / esize;
            c.ub = chunk + (aligned ? 0 : 16);
            c.batch = std::min(c.nsrc, rows_part(c.nsrc) / (SP_GROUPS * c.ub));
            const u64 chunks = (c.nu + c.per - 1) / c.per;
            c.rows = (u32)std::min((double)chunks, SP_WARPS * std::max(1.0, target / (row * chunk * SP_WARPS)));
            if (lone) {
                // two tiles for each SM, or four where each folds many sources in a short
                // call (two / four: 16 ranks of 500001 int32 16.0 / 14.0 us, of 1562497
                // 38.5 / 43.5; Reduce of 64 of 390625 33.5 / 30.1)
                const u32 k = c.nsrc < 16 || (c.nsrc < 32 && total >= 1e8) ? 2 : 4;
                c.rows = (u32)round_up(split(chunks, k * SP_SMS), SP_WARPS);
            }
            if (lone && many) c.rows = (u32)split(chunks, 4 * SP_SMS);
            // a large call: equal tiles in whole waves, at most a chunk for each warp (chunks
            // that are halved until they make three tiles for each block, as among other
            // calls / so, us: Reduce of FP64, 256 ranks of 126952 132 / 81, of 195312 226 /
            // 119, 320 of 156248 202 / 124, 64 of 1562501 229 / 209; Allreduce of 256 of 97656
            // 172 / 96; the rank blocks took 121, 156, 186, 480 and 152)
            if (large && c.nsrc >= 16) c.rows = (u32)split(chunks, 4 * SP_SMS * split(chunks, 4 * SP_SMS * SP_WARPS));
            if (passes) c.rows = 1;
            c.ntiles = (u32)((chunks + c.rows - 1) / c.rows);
            c.tile_bytes = (u32)(row * chunk * c.rows);
            calls.push_back(c);
            if (lo) gather(0, 2 * lo, lo, n - lo);
            else if (hi < n) gather(hi, n - hi, n - hi, n - hi);
            return;
        }
        if (lone) {
            // two whole waves rather than one and a bit, unless that halves the warps'
            // additions too (64 ranks of 62496 FP64, 100 elements 21.4, 52 18.7 us; 200
            // of 124992 float32, 64 elements 40.4, 52 44.5 us)
            const u64 m = round_up(split(n, 8 * SP_SMS), step);
            const u64 per = m >= 48 && m <= most ? m : most;
            gather_all(per);
            return;
        }
        // A warp's addition takes the same time however many lanes add: fill it as
        // far as that leaves two tiles for each block (the 16-communicator batch at
        // 301 per rank 20.7 -> 18.2 us, at 1024 28.7 -> 23.4 us)
        const double fill = std::min(32.0, std::ceil(level.folded / (SP_SMS * SP_BLOCKS_PER_SM * 2)));
        const double per = std::min(fits, std::max(target / 2 / ((double)P * esize), fill));
        const u64 m = std::max(step, (u64)std::min(per, (double)n) / step * step);
        gather_all(m);
        return;
    }
    const bool a2a = d.op == GPUMPI_COLL_ALLTOALL;
    c.rs = a2a ? bytes : 0;
    // The end alone of a Bcast's block would make its units 1 or 2 bytes: it goes as a
    // gather tile of one source (uint8 to 128 ranks, rank blocks / with its own units /
    // so, us: 600001 elements 21 / 26 / 15, 2400001 60 / 164 / 56; to 256 ranks 35 / 83 /
    // 35, 107 / 326 / 104; 10001 to 64 ranks 6.2 / 4.1 / 2.6).
    if (c.nsrc == 1 && bits % 16 == 0 && bytes % 4 && bytes >= RAGGED_BYTES) {
        SpreadCall end = c;
        end.kind = SP_GATHER;
        end.fn = (esize == 1 ? FT_I8 : FT_I16) * 4 + GPUMPI_OP_MAX;
        end.off = bytes / 16 * 16;
        end.nu = bytes % 16 / esize;
        end.per = (u32)end.nu;
        end.rs = 0;
        end.ub = esize;
        end.ntiles = 1;
        end.tile_bytes = (u32)((1 + c.ndst) * (bytes % 16));
        calls.push_back(end);
        bytes = end.off;
    }
    bits |= bytes;
    const bool units16 = bits % 16 == 0;
    c.ub = units16 ? 16 : bits % 8 == 0 ? 8 : bits % 4 == 0 ? 4 : bits % 2 == 0 ? 2 : 1;
    const u64 move_min = c.ub >= 4 ? SP_MOVE_UNITS : move_bytes(c.ub, (u64)c.nsrc * c.ndst);
    bool move = bytes >= (a2a ? move_min : fan_min(units16, total));
    bool fan = !a2a && bytes / c.ub >= 2 * SP_T, halves = false;
    // SP_COPY by chunks, where at most a quarter of the lanes' turns is empty: for
    // 4-byte units (int32 Alltoall of the 16 communicators, 30001 per rank 73.9 ->
    // 53.4 us, 100003 182 -> 160; the whole batch at 50000 511 -> 505) and lone calls
    // of 8-byte units (16 ranks, 64 MB 13.2 -> 8.7 us, but FP64 Alltoall of all 16
    // communicators at 100003 284 -> 296).  16-byte units gain nothing (64 MB 9.4,
    // 10.1), nor do shorter blocks among other calls (the batch at 301 17.3, 17.6 us).
    const u64 units = bytes / c.ub;
    const bool chunks = units >= (lone ? 1 : 4 * SP_CHUNK) && (c.ub == 4 || (lone && c.ub == 8)) &&
                        round_up(units, SP_CHUNK) * 3 <= units * 4;
    u32 even = 2 * SP_SMS;   // tiles of a lone call
    if (lone && a2a) {
        // The deep ring of a few long SP_COPY tiles beats bulk copies for units of 4
        // bytes and more (64 ranks, SP_COPY / SP_MOVE: 16-byte units, 16 MB 4.1 / 8.1 us,
        // 64 MB 8.6 / 14.3; 8-byte units 200 MB 40 / 45; 4-byte units 64 MB 11.1 / 17.1, 200
        // MB 41 / 45), unless 4-byte units have to go one at a time (64 MB 23.8 / 17.1)
        move = bytes >= move_bytes(c.ub, (u64)c.nsrc * c.ndst) && (c.ub < 4 || (c.ub == 4 && !chunks && total >= 8e6));
        if (move) even = total < 4e6 ? SP_SMS : total < 3e7 ? 2 * SP_SMS : 4 * SP_SMS;
    } else if (large && a2a && c.ub == 16) {
        // The same holds for 16-byte units of larger calls, in tiles of 128 KiB (FP64, 128
        // ranks, SP_MOVE / SP_COPY: 400 MB 90 / 68 us, 1.6 GB 281 / 252, 4 GB 666 / 622; 200
        // ranks, 4 GB 670 / 641; tiles of 300 KB 71, 259, 638, of 2 MB 78, 298, 632).
        // Rank blocks took 254 and 606 us for the second and the third.
        move = false;
    } else if (lone) {
        // Bulk copies need the call to be large and a few hundred pieces (Allgather of
        // 64 ranks, 100 MB: SP_MOVE 18.1, SP_FAN 26, SP_COPY 23.5 us; 32 MB 8.7, 9.0, 8.6;
        // Bcast of 500 KB to 200 ranks, 80 pieces: 26, 20.8, 23).  SP_FAN reads a unit
        // once for several destinations, which pays once the stores no longer fit the
        // same few tiles (Bcast of 16-byte units to 16 ranks, SP_FAN / SP_COPY: 8 MB 6.1 /
        // 4.0 us, 32 MB 7.6 / 8.3; of 8-byte units 8 MB 3.6 / 5.2, 32 MB 7.0 / 12.6).
        // (From 160 MB a Bcast of fewer goes in pieces of half the length: 200 ranks of
        // 900000 bytes SP_FAN 37.4, SP_MOVE 29.6, half 29.8; of 1225000 49.0, 44.4, 39.6; 256
        // of 957024 58.3, 54.5, 42.3; 512 of 410144 49.1, 48.0, 34.3; rank blocks 256 of
        // 957024 49 us.)
        move = total >= 8e7 && bytes >= 2048 && split(bytes, SP_FAN_PIECE) * c.nsrc >= 200;
        halves = !move && units16 && c.nsrc == 1 && total >= 1.6e8;
        move = move || halves;
        fan = fan && (!units16 || total >= 1.6e7);
        if (move && units16) even = SP_SMS;
    }
    if (move) {
        // a large call has warps enough for one long row each (Alltoall of odd FP64 buffers,
        // pieces of 1920 / 6016 bytes: 128 ranks, 800 MB 165 / 150, 4 GB 722 / 646 us)
        const u64 longest = a2a && !large ? SP_PIECE : halves ? SP_HALF_PIECE : SP_FAN_PIECE;
        c.kind = SP_MOVE;
        c.cold = total >= 1e8;
        c.nu = bytes;
        const u64 pieces = (bytes + longest - 1) / longest;
        const u64 step = pieces > 1 ? 128 : 16;
        c.per = (u32)(((bytes + pieces - 1) / pieces + step - 1) / step * step);
        c.stages = std::min((u32)SP_MAX_STAGES, SP_PART / (c.per + 32));
        const double sets = units16 ? SP_FAN_ALIGNED : SP_FAN_ODD;
        const double stored = lone ? total / even : target;
        c.group = a2a ? 1 : (u32)std::min((double)c.ndst, std::max(1.0, std::min(sets, stored / c.per)));
        const u64 rows = (bytes + c.per - 1) / c.per * c.nsrc * ((c.ndst + c.group - 1) / c.group);
        // at least a row for each warp (8 ranks of 2^17 FP64 11.8 -> 7.4 us)
        c.rows = (u32)std::max(a2a ? (double)SP_WARPS : 1.0, target / ((1.0 + c.group) * c.per));
        if (lone) c.rows = (u32)split(rows, even);
        c.ntiles = (u32)((rows + c.rows - 1) / c.rows);
        calls.push_back(c);
        return;
    }
    c.nu = bytes / c.ub;
    if (fan) {
        c.kind = SP_FAN;
        // (shorter calls and larger ones of small units are better off with the sizes
        // below: Bcast of 8-byte units, 2 MB 2.9 against 3.2 us; of 4-byte units to 200
        // ranks, 100 MB 23.7 against 27.6)
        if (lone && total >= 4e6 && (units16 || total < 8e7)) {
            // The least that the SM with most tiles moves, a tile's start counting as
            // 20000 bytes (Bcast of 32 MB to 64 ranks, 275 tiles 7.2, 325 tiles 11.3 us)
            double best = 1e30;
            for (u32 g = 1; g <= std::min(c.ndst, 16u); g++)
                for (u64 k = 1; k <= 16; k++) {
                    const u64 per = std::min(k * SP_T, round_up(c.nu, SP_T));
                    const u64 tiles = split(c.nu, per) * c.nsrc * split(c.ndst, g);
                    const double tile = 20000.0 + (double)std::min(per, c.nu) * c.ub * (g + 1);
                    const double cost = (double)split(tiles, SP_SMS) * tile;
                    if (cost >= best) continue;
                    best = cost;
                    c.group = g;
                    c.per = (u32)per;
                    c.ntiles = (u32)tiles;
                }
            calls.push_back(c);
            return;
        }
        // a tile stores 64 KiB and more (256 KiB when the launch is large) to 4 to 8
        // destinations, less only to give every SM a tile
        const double stored = std::min(262144.0, std::max(65536.0, target));
        u64 per = c.ub == 16 && target < 262144.0 ? 4 * SP_T : 8 * SP_T;
        const double sets = std::min(8.0, std::max(4.0, stored / ((double)per * c.ub)));
        c.group = (u32)std::min((double)c.ndst, sets);
        while (per > 2 * SP_T && (double)c.nu * c.nsrc * c.ndst < (double)SP_SMS * per * c.group) per /= 2;
        const u64 pieces = (c.nu + per - 1) / per;
        per = ((c.nu + pieces - 1) / pieces + SP_T - 1) / SP_T * SP_T;
        c.per = (u32)per;
        c.ntiles = (u32)((c.nu + per - 1) / per * c.nsrc * ((c.ndst + c.group - 1) / c.group));
    } else {
        c.kind = SP_COPY;
        c.group = chunks;
        const u64 item = c.group ? SP_CHUNK : 1, step = SP_T / 32 * (c.group ? 1 : 32);
        const u64 items = (u64)c.ndst * c.nsrc * split(units, item);
        u64 per = step * (u64)std::max(1.0, target / (2.0 * step * item * c.ub));
        if (lone) per = round_up(split(items, even), step);
        if (large && a2a && c.ub == 16) per = 4096;
        c.per = (u32)per;
        c.ntiles = (u32)split(items, per);
    }
    calls.push_back(c);
}

// Bytes that a tile moves.
static double tile_cost(const SpreadCall& c) {
    switch (c.kind) {
        case SP_FAN: return (double)c.per * c.ub * (1 + c.group);
        case SP_COPY: return 2.0 * c.per * c.ub * (c.group ? SP_CHUNK : 1);
        case SP_MOVE: return (1.0 + c.group) * c.rows * c.per;
        default: return (double)c.tile_bytes;
    }
}

void SpreadBuilder::end_level() {
    SpreadLevel l = {};
    l.first_call = levels.empty() ? 0 : levels.back().first_call + levels.back().ncalls;
    l.ncalls = (u32)calls.size() - l.first_call;
    // the longest tiles first: one that starts last would run alone
    std::stable_sort(calls.begin() + l.first_call, calls.end(), [](const SpreadCall& a, const SpreadCall& b) {
        return tile_cost(a) > tile_cost(b);
    });
    for (u32 i = l.first_call; i < (u32)calls.size(); i++) {
        calls[i].first_tile = l.ntiles;
        l.ntiles += calls[i].ntiles;
    }
    levels.push_back(l);
}

bool SpreadBuilder::params(SpreadParams* p) const {
    if (calls.size() > SP_PARAM_CALLS || ptrs.size() > 2 * SP_PARAM_RANKS || levels.size() != 1) return false;
    std::copy(calls.begin(), calls.end(), p->calls);
    std::copy(ptrs.begin(), ptrs.end(), p->ptrs);
    p->ncalls = (u32)calls.size();
    p->ntiles = levels[0].ntiles;
    return true;
}

size_t SpreadBuilder::bytes() const { return sizeof(SpreadCall) * calls.size() + sizeof(void*) * ptrs.size(); }

size_t SpreadBuilder::max_bytes(int nranks) {
    return sizeof(SpreadCall) * SP_PARAM_CALLS + sizeof(void*) * 2 * (size_t)nranks;
}

void SpreadBuilder::image(char* host, char* dev, SpreadArgs* args) {
    const size_t ptrs_at = sizeof(SpreadCall) * calls.size();
    for (SpreadCall& c : calls) {
        c.src = (const char* const*)(dev + ptrs_at + (size_t)c.src * sizeof(void*));
        c.dst = (char* const*)(dev + ptrs_at + (size_t)c.dst * sizeof(void*));
    }
    if (!calls.empty()) {
        memcpy(host, calls.data(), sizeof(SpreadCall) * calls.size());
        memcpy(host + ptrs_at, ptrs.data(), sizeof(void*) * ptrs.size());
    }
    for (size_t l = 0; l < levels.size(); l++) {
        SpreadArgs& a = args[l];
        memset(&a, 0, sizeof(a));
        if (levels[l].ncalls) a.one = calls[levels[l].first_call];
        a.calls = (const SpreadCall*)dev + levels[l].first_call;
        a.ncalls = levels[l].ncalls;
        a.ntiles = levels[l].ntiles;
    }
}

}  // namespace gm
