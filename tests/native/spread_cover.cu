// CPU emulation of tile lists (csrc/spread.cuh) for calls of up to SP_MAX_RANKS
// ranks: every tile's reads lie inside the source buffers, its shared memory
// inside the block's, and what all tiles write covers each destination buffer
// exactly once, without a gap or an overlap.  Random calls with seed SEED, or
// one named call (for the kind of tile that its sizes are meant to reach).
// Prints the forms of tiles seen.
// Usage: spread_cover random SEED CALLS
//        spread_cover one OP RANKS COUNT DTYPE ELEMENT_SIZE SKEW [LEVEL_CALLS LEVEL_BYTES]
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <string>
#include <vector>

#include "spread.cuh"
using namespace gm;

static long bad = 0;
static std::string call_text;
#define CHECK(x)                                                               \
    do {                                                                       \
        if (!(x) && bad++ < 20) printf("BAD %s: %s\n", #x, call_text.c_str()); \
    } while (0)

struct Buffer {
    u64 at, bytes;
};
struct Range {
    u64 lo, hi;
};

// The accesses of one tile list.
struct Tiles {
    const SpreadBuilder& b;
    const std::vector<Buffer>& src;   // by source number
    int es;
    std::map<u64, std::vector<Range>> written;   // by destination address
    std::map<std::string, long> forms;

    u64 from(const SpreadCall& c, u64 q) {
        CHECK(q < c.nsrc);
        return (u64)b.ptrs[(size_t)c.src + q];
    }
    void read(const SpreadCall& c, u64 q, u64 at, u64 n) {
        CHECK(from(c, q) == src[q].at);
        CHECK(at >= src[q].at && at + n <= src[q].at + src[q].bytes);
    }
    // `off` bytes into destination r
    void write(const SpreadCall& c, u64 r, u64 off, u64 n) {
        CHECK(r < c.ndst && n > 0);
        written[(u64)b.ptrs[(size_t)c.dst + r]].push_back({off, off + n});
    }
    void write_all(const SpreadCall& c, u64 off, u64 n) {
        for (u64 r = 0; r < c.ndst; r++) write(c, r, off, n);
    }

    void fan(const SpreadCall& c, u64 t) {
        const u64 pieces = (c.nu + c.per - 1) / c.per, q = t / pieces % c.nsrc;
        const u64 r0 = t / pieces / c.nsrc * c.group, r1 = std::min<u64>(r0 + c.group, c.ndst);
        const u64 o0 = t % pieces * c.per, o1 = std::min<u64>(o0 + c.per, c.nu);
        CHECK(r0 < c.ndst && from(c, q) % c.ub == 0);
        read(c, q, from(c, q) + o0 * c.ub, (o1 - o0) * c.ub);
        for (u64 r = r0; r < r1; r++) write(c, r, (q * c.nu + o0) * c.ub, (o1 - o0) * c.ub);
    }
    void copy(const SpreadCall& c, u64 t) {
        const u64 item = c.group ? SP_CHUNK : 1, len = (c.nu + item - 1) / item;
        const u64 total = (u64)c.ndst * c.nsrc * len, k1 = std::min<u64>((t + 1) * c.per, total);
        CHECK(t * c.per < total && c.nu < (1ull << 32) && (!c.group || c.ub >= 4));
        for (u64 k = t * c.per; k < k1; k++) {
            const u64 q = k / len % c.nsrc, r = k / len / c.nsrc, o = k % len * item, n = std::min(item, c.nu - o);
            const u64 at = from(c, q) + c.rs * r + o * c.ub;
            CHECK(at % c.ub == 0);
            read(c, q, at, n * c.ub);
            write(c, r, (q * c.nu + o) * c.ub, n * c.ub);
        }
    }
    void gather(const SpreadCall& c, u64 t) {
        const u64 m = std::min<u64>(c.per, c.nu - t * c.per), at = c.off + t * c.rs;
        CHECK(t * c.per < c.nu && m * es * c.nsrc <= SP_RING);
        CHECK(c.ub == 16 ? m * es % 16 == 0 : (int)c.ub == es);
        for (u64 q = 0; q < c.nsrc; q++) {
            CHECK((from(c, q) + at) % c.ub == 0);
            read(c, q, from(c, q) + at, m * es);
        }
        write_all(c, at, m * es);
    }
    void stream(const SpreadCall& c, u64 t) {
        const u64 nvec = c.nu * es / 16, v0 = t * c.per * SP_T, v1 = std::min<u64>(nvec, v0 + (u64)c.per * SP_T);
        CHECK(v0 < nvec && c.nsrc <= SP_TAB);
        for (u64 q = 0; q < c.nsrc; q++) {
            CHECK((from(c, q) + c.off) % 16 == 0);
            read(c, q, from(c, q) + c.off + v0 * 16, (v1 - v0) * 16);
        }
        write_all(c, c.off + v0 * 16, (v1 - v0) * 16);
    }
    // a chunk folded by the whole block
    void passes(const SpreadCall& c, u64 t) {
        const u64 m = std::min<u64>(c.per, c.nu - t * c.per), at = c.off + t * c.per * es;
        const u64 half = passes_half(c.nsrc), batch = half / (c.per * es), unit = c.ub == c.per * es ? 16 : es;
        CHECK(t * c.per < c.nu && c.rows == 1 && c.per <= SP_T && batch >= 1);
        CHECK(2 * half <= fold_table(c.nsrc) && half % 16 == 0 && fold_table(c.nsrc) + 8 * c.nsrc <= SP_SMEM);
        CHECK(SP_T * es + 8ull * c.ndst <= fold_table(c.nsrc) && batch * m * es <= half && m * es % unit == 0);
        for (u64 q = 0; q < c.nsrc; q++) {
            CHECK((from(c, q) + at) % unit == 0);
            read(c, q, from(c, q) + at, m * es);
        }
        write_all(c, at, m * es);
    }
    void rows(const SpreadCall& c, u64 t) {
        const u64 all = (c.nu + c.per - 1) / c.per, w1 = std::min<u64>((t + 1) * c.rows, all), part = rows_part(c.nsrc);
        CHECK(t * c.rows < all && c.batch >= 1 && c.batch * c.ub * 3 <= part && c.per * es <= 512 && c.per % 32 == 0);
        CHECK(part % 16 == 0 && part * SP_WARPS <= (c.nsrc > SP_TAB ? fold_table(c.nsrc) : SP_RING));
        for (u64 w = t * c.rows; w < w1; w++) {
            const u64 m = std::min<u64>(c.per, c.nu - w * c.per), at = c.off + w * c.per * es;
            for (u64 q = 0; q < c.nsrc; q++) {
                const u64 x = from(c, q) + at, x0 = x & ~15ull, x1 = (x + m * es + 15) & ~15ull;
                CHECK(x1 - x0 <= c.ub);
                read(c, q, x0, x1 - x0);
            }
            write_all(c, at, m * es);
        }
    }
    void move(const SpreadCall& c, u64 t) {
        const u64 pieces = (c.nu + c.per - 1) / c.per, sets = (c.ndst + c.group - 1) / c.group;
        const u64 all = pieces * c.nsrc * sets, extent = c.rs ? c.rs * c.ndst : c.nu;
        CHECK(t * c.rows < all && all < (1ull << 32) && c.stages >= 1 && c.stages <= SP_MAX_STAGES);
        CHECK(c.stages * (c.per + 32) <= SP_PART && c.per % 16 == 0);
        for (u64 row = t * c.rows; row < std::min<u64>((t + 1) * c.rows, all); row++) {
            u64 piece, q, r0;
            if (c.rs) {
                piece = row % pieces, q = row / pieces % c.nsrc, r0 = row / pieces / c.nsrc;
            } else {
                r0 = row % sets * c.group, piece = row / sets % pieces, q = row / sets / pieces;
            }
            const u64 p0 = piece * c.per, len = std::min<u64>(c.per, c.nu - p0), off = c.rs * r0 + p0;
            const u64 a = from(c, q) + off, e = a + len;
            const u64 x0 = off >= 16 ? a & ~15ull : (a + 15) & ~15ull;
            const u64 x1 = off + len + 16 <= extent ? (e + 15) & ~15ull : e & ~15ull;
            read(c, q, a, len);
            if (x1 > x0) read(c, q, x0, x1 - x0);
            CHECK(x1 <= x0 || x1 - x0 <= c.per + 32);
            for (u64 r = r0; r < (c.rs ? r0 + 1 : std::min<u64>(r0 + c.group, c.ndst)); r++)
                write(c, r, q * c.nu + p0, len);
        }
    }
    void run() {
        u64 next = 0;
        for (const SpreadCall& c : b.calls) {
            CHECK(c.first_tile == next && c.ntiles > 0);
            next += c.ntiles;
            static const char* const names[] = {"fan", "copy", "gather", "stream", "move", "rows"};
            std::string form = names[c.kind];
            if (c.kind == SP_COPY && c.group) form = "chunks";
            if (c.kind == SP_ROWS) form = c.group ? "passes" : c.nsrc > SP_TAB ? "rows-many" : "rows";
            if (c.kind == SP_MOVE) form = c.rs ? "move-alltoall" : "move-fan";
            forms[form] += c.ntiles;
            for (u32 t = 0; t < c.ntiles; t++) switch (c.kind) {
                    case SP_FAN: fan(c, t); break;
                    case SP_COPY: copy(c, t); break;
                    case SP_GATHER: gather(c, t); break;
                    case SP_STREAM: stream(c, t); break;
                    case SP_MOVE: move(c, t); break;
                    default:
                        if (c.group) passes(c, t);
                        else rows(c, t);
                }
        }
        CHECK(next == b.levels[0].ntiles);
    }
};

static std::map<std::string, long> seen;

// One call, as part of a level that it makes up by itself unless `calls` and `bytes` are given.
static void check(int op, int P, u64 n, int dtype, int es, int skew, int calls, double bytes, long max_tiles) {
    char text[200];
    snprintf(text, sizeof(text), "op %d ranks %d count %llu dtype %d skew %d calls %d bytes %.0f", op, P, n, dtype, skew,
             calls, bytes);
    call_text = text;
    const u64 slen = (op == GPUMPI_COLL_ALLTOALL ? n * P : n) * es, rlen = (op >= GPUMPI_COLL_ALLTOALL ? n * P : n) * es;
    std::vector<void*> s(P), r(P);
    std::vector<Buffer> sb(P), rb(P);
    u64 at = 0x10000000;
    auto place = [&](void*& p, Buffer& buf, u64 len, int step) {
        buf = {at + (skew ? (u64)step * skew * es % 16 : 0), len};
        p = (void*)buf.at;
        at = (buf.at + len + 300) / 16 * 16;
    };
    for (int i = 0; i < P; i++) place(s[i], sb[i], slen, i);
    for (int i = 0; i < P; i++) place(r[i], rb[i], rlen, 3 * i);
    gpumpi_coll_desc d;
    memset(&d, 0, sizeof(d));
    d.op = op;
    d.dtype = dtype;
    d.redop = GPUMPI_OP_MAX;
    d.root = (int)(n % P);
    d.count = n;
    d.sendbufs = op == GPUMPI_COLL_BCAST ? nullptr : s.data();
    d.recvbufs = r.data();
    if (!SpreadBuilder::covers(d, P, es)) {
        CHECK(!"covered");
        return;
    }
    SpreadLoad level;
    level.count(d, P, es);
    if (calls > 1) {
        level.calls = calls;
        level.folded *= std::max(1.0, bytes / level.bytes);
        level.bytes = std::max(level.bytes, bytes);
    }
    SpreadBuilder b;
    b.add(d, P, es, level);
    b.end_level();
    if (max_tiles && b.levels[0].ntiles > max_tiles) return;
    std::vector<Buffer> src = sb;
    if (op == GPUMPI_COLL_BCAST) src.assign(1, rb[d.root]);
    Tiles tiles{b, src, es, {}, {}};
    tiles.run();
    for (auto& f : tiles.forms) seen[f.first] += f.second;
    for (int i = 0; i < P; i++) {
        std::vector<Range>& w = tiles.written[rb[i].at];
        std::sort(w.begin(), w.end(), [](const Range& x, const Range& y) { return x.lo < y.lo; });
        u64 end = 0;
        for (const Range& x : w) {
            CHECK(x.lo == end);
            end = x.hi;
        }
        const bool other = (op == GPUMPI_COLL_BCAST && i == d.root) || (op == GPUMPI_COLL_REDUCE && i != d.root);
        CHECK(end == (other ? 0 : rlen));
    }
    // above SP_TAB ranks no fold leaves most of a warp's lanes without an element for more
    // than two tiles for each block (FP64 additions cost the same for 2 lanes as for 32)
    if (P > SP_TAB && (op == GPUMPI_COLL_REDUCE || op == GPUMPI_COLL_ALLREDUCE) && es > 1)
        for (const SpreadCall& c : b.calls) CHECK(c.kind != SP_GATHER || c.per >= 32 || c.ntiles <= 2 * 4 * 152);
    // whole buffers of 1- and 2-byte elements on 16-byte boundaries do not go element by
    // element, whatever their length: at most their last 15 bytes do
    const bool fold = op == GPUMPI_COLL_REDUCE || op == GPUMPI_COLL_ALLREDUCE;
    if (skew == 0 && es < 4 && fold && n >= 1024)
        for (const SpreadCall& c : b.calls) CHECK(c.kind != SP_GATHER || c.ub == 16 || c.nu * es < 16);
    if (skew == 0 && es < 4 && op == GPUMPI_COLL_BCAST && n * es >= 4096)
        for (const SpreadCall& c : b.calls) CHECK((c.kind != SP_FAN && c.kind != SP_COPY) || c.ub >= 4);
}

int main(int argc, char** argv) {
    auto arg = [&](int i) { return i < argc ? atof(argv[i]) : 0.0; };
    if (std::string(argv[1]) == "one") {
        check((int)arg(2), (int)arg(3), (u64)arg(4), (int)arg(5), (int)arg(6), (int)arg(7), (int)arg(8), arg(9), 0);
    } else {
        std::mt19937_64 rng((u64)arg(2));
        auto uniform = [&](u64 lo, u64 hi) { return lo + rng() % (hi - lo + 1); };
        auto spread = [&](double lo, double hi) { return (u64)(lo * pow(hi / lo, (double)(rng() % 100000) / 1e5)); };
        static const int types[] = {6, 1, 2, 13, 12, 29, 20}, sizes[] = {1, 2, 4, 8, 4, 1, 8};
        for (int i = 0; i < (int)arg(3); i++) {
            const int op = (int)uniform(1, 5), k = (int)uniform(0, 6);
            const int P = (int)(i % 4 ? spread(1, 64) : spread(200, SP_MAX_RANKS));
            const u64 n = spread(1, 8e6 / P / (op >= 4 ? P : 1) + 2);
            const bool among = i % 3 == 0;
            check(op, P, n, types[k], sizes[k], (int)uniform(0, 3), among ? 5 : 1, among ? spread(1e4, 4e9) : 0, 2500);
        }
    }
    printf("bad %ld forms", bad);
    for (auto& f : seen) printf(" %s", f.first.c_str());
    printf("\n");
    return bad != 0;
}
