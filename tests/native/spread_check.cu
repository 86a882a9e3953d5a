// CPU emulation of the tiles of the spread form (csrc/spread.cuh): for random
// calls of every collective, element size, rank count, length and alignment, in
// levels of many sizes, every tile's reads lie inside the source buffers, every
// destination byte is written exactly once, alignments are those its copies
// need and its rows fit the ring.  Prints the tiles seen and what was wrong.
// Usage: spread_check SEED CALLS
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <cmath>
#include <map>
#include <random>
#include "spread.cuh"
using namespace gm;
static long bad = 0;
#define CHK(x, ...) do { if (!(x)) { if (bad++ < 20) { printf("BAD %s:", #x); printf(__VA_ARGS__); printf("\n"); } } } while (0)
struct Buf { u64 a, n; };
static bool in(const Buf& b, u64 a, u64 n) { return a >= b.a && a + n <= b.a + b.n; }
int main(int argc, char** argv) {
    std::mt19937_64 rng(atoi(argv[1]));
    auto R = [&](u64 lo, u64 hi) { return lo + rng() % (hi - lo + 1); };
    auto L = [&](double lo, double hi) { return (u64)(lo * pow(hi / lo, (rng() % 100000) / 1e5)); };
    long tiles = 0; std::map<int, long> kinds;
    for (int it = 0; it < atoi(argv[2]); it++) {
        int P = (int)L(1, it % 10 == 0 ? 600 : 64), op = (int)R(1, 5);
        static const int DT[] = {6, 1, 2, 13, 12, 29, 20}; static const int ES[] = {1, 2, 4, 8, 4, 1, 8};
        int k = (int)R(0, 6), es = ES[k];
        u64 n = L(1, 4e6 / P / (op >= 4 ? P : 1) + 2);
        int skew = (int)R(0, 3);
        u64 sl = op == 4 ? n * P : n, rl = op >= 4 ? n * P : n;
        std::vector<void*> s(P), r(P); std::vector<Buf> sb(P), rb(P);
        u64 a = 0x10000000;
        for (int i = 0; i < P; i++) { u64 x = a + (skew ? (i * skew * es) % 16 : 0); s[i] = (void*)x; sb[i] = {x, sl * es}; a = (x + sl * es + 300) / 16 * 16; }
        for (int i = 0; i < P; i++) { u64 x = a + (skew ? (i * skew * es * 3) % 16 : 0); r[i] = (void*)x; rb[i] = {x, rl * es}; a = (x + rl * es + 300) / 16 * 16; }
        gpumpi_coll_desc d; memset(&d, 0, sizeof d); d.op = op; d.dtype = DT[k]; d.redop = (int)R(0, 3); d.root = (int)R(0, P - 1); d.count = n;
        d.sendbufs = op == 1 ? nullptr : s.data(); d.recvbufs = r.data();
        if (!SpreadBuilder::covers(d, P, es)) continue;
        SpreadLoad lv; lv.count(d, P, es);
        if (it % 3 == 0) { lv.calls = 2; lv.bytes *= R(1, 200); lv.folded *= R(1, 200); }   // one of several calls of its level
        if (it % 3 == 1) lv.bytes *= R(1, 30);   // the choices of larger calls
        SpreadBuilder b; b.add(d, P, es, lv); b.end_level();
        if (b.levels[0].ntiles > 3000) continue;
        std::vector<Buf> src, dst;
        if (op == 1) src.push_back(rb[d.root]); else src = sb;
        std::map<u64, long> wrote;   // destination bytes written, by buffer
        for (auto& c : b.calls) {
            auto ps = [&](u64 q) { CHK(q < c.nsrc, "q %llu nsrc %u", q, c.nsrc); return (u64)b.ptrs[(size_t)c.src + q]; };
            auto pd = [&](u64 q) { CHK(q < c.ndst, "r %llu ndst %u", q, c.ndst); return (u64)b.ptrs[(size_t)c.dst + q]; };
            auto rd = [&](u64 q, u64 x, u64 m) { const Buf& f = op == 1 ? rb[d.root] : sb[q]; CHK(in(f, x, m), "read kind %d op %d P %d n %llu es %d q %llu off %lld m %llu of %llu", c.kind, op, P, n, es, q, (long long)(x - f.a), m, f.n); };
            auto wr = [&](u64 p, u64 x, u64 m) { int i = -1; for (int j = 0; j < P; j++) if (rb[j].a == p) i = j; CHK(i >= 0 && in(rb[i], x, m), "write kind %d op %d P %d n %llu es %d", c.kind, op, P, n, es); wrote[p] += m; };
            tiles += c.ntiles; kinds[c.kind] += c.ntiles;
            CHK(c.first_tile + c.ntiles <= b.levels[0].ntiles, "tiles");
            for (u32 t = 0; t < c.ntiles; t++) {
                if (c.kind == SP_COPY) {
                    // items: units, or chunks of SP_CHUNK units of one block
                    CHK(c.nu < (1ull << 32) && (!c.group || c.ub >= 4), "nu");
                    u64 item = c.group ? SP_CHUNK : 1, len = (c.nu + item - 1) / item;
                    u64 total = (u64)c.ndst * c.nsrc * len, k1 = std::min<u64>((u64)(t + 1) * c.per, total);
                    CHK((u64)t * c.per < total, "empty tile");
                    for (u64 k = (u64)t * c.per; k < k1; k++) {
                        u64 blk = k / len, o = k % len * item, m = std::min(item, c.nu - o), rr = blk / c.nsrc, q = blk % c.nsrc;
                        u64 from = ps(q) + c.rs * rr + o * c.ub, to = pd(rr) + (q * c.nu + o) * c.ub;
                        rd(q, from, m * c.ub); CHK(from % c.ub == 0 && to % c.ub == 0, "align"); wr(pd(rr), to, m * c.ub);
                    }
                } else if (c.kind == SP_FAN) {
                    u32 pieces = (u32)((c.nu + c.per - 1) / c.per), piece = t % pieces, rest = t / pieces; u64 q = rest % c.nsrc, r0 = (u64)rest / c.nsrc * c.group, r1 = std::min<u64>(r0 + c.group, c.ndst), o0 = (u64)piece * c.per, o1 = std::min<u64>(o0 + c.per, c.nu);
                    CHK(r0 < c.ndst, "r0"); rd(q, ps(q) + c.rs * r0 + o0 * c.ub, (o1 - o0) * c.ub);
                    for (u64 x = r0; x < r1; x++) wr(pd(x), pd(x) + (q * c.nu + o0) * c.ub, (o1 - o0) * c.ub);
                } else if (c.kind == SP_GATHER) {
                    CHK((u64)t * c.per < c.nu, "empty tile"); u64 m = std::min<u64>(c.per, c.nu - (u64)t * c.per), at = c.off + t * c.rs; CHK(m * es * c.nsrc <= SP_RING, "ring m %llu P %d es %d", m, P, es);
                    CHK(c.ub == 16 ? m * es % 16 == 0 : (int)c.ub == es, "ub");
                    for (u32 q = 0; q < c.nsrc; q++) { rd(q, ps(q) + at, m * es); CHK((ps(q) + at) % c.ub == 0, "align"); }
                    for (u32 x = 0; x < c.ndst; x++) { wr(pd(x), pd(x) + at, m * es); CHK((pd(x) + at) % c.ub == 0, "align"); }
                } else if (c.kind == SP_STREAM) {
                    u64 nvec = c.nu * es / 16, v0 = (u64)t * c.per * SP_T; CHK(v0 < nvec, "empty"); u64 v1 = std::min<u64>(nvec, v0 + (u64)c.per * SP_T);
                    for (u32 q = 0; q < c.nsrc; q++) { rd(q, ps(q) + c.off + v0 * 16, (v1 - v0) * 16); CHK((ps(q) + c.off) % 16 == 0, "align"); }
                    for (u32 x = 0; x < c.ndst; x++) wr(pd(x), pd(x) + c.off + v0 * 16, (v1 - v0) * 16);
                } else if (c.kind == SP_ROWS) {
                    u64 all = (c.nu + c.per - 1) / c.per, w0 = (u64)t * c.rows, w1 = std::min<u64>(w0 + c.rows, all); CHK(w0 < all, "empty");
                    CHK(c.batch >= 1 && c.batch * c.ub * 3 <= SP_PART && c.ub % 16 == 0, "part"); CHK(c.per * es <= 512 && c.per % 32 == 0, "per");
                    for (u64 w = w0; w < w1; w++) { u64 e0 = w * c.per, m = std::min<u64>(c.per, c.nu - e0), at = c.off + e0 * es;
                        for (u32 q = 0; q < c.nsrc; q++) { u64 x = ps(q) + at, x0 = x & ~15ull, x1 = (x + m * es + 15) & ~15ull; rd(q, x0, x1 - x0); CHK((x & 15) + m * es <= c.ub && x1 - x0 <= c.ub, "pitch"); }
                        for (u32 y = 0; y < c.ndst; y++) wr(pd(y), pd(y) + at, m * es); }
                } else if (c.kind == SP_MOVE) {
                    u64 pieces = (c.nu + c.per - 1) / c.per, sets = (c.ndst + c.group - 1) / c.group, all = pieces * c.nsrc * sets; u64 row0 = (u64)t * c.rows, row1 = std::min<u64>(row0 + c.rows, all); CHK(row0 < all, "empty"); CHK(all < (1ull << 32), "rows");
                    CHK(c.stages >= 1 && c.stages <= 8 && c.stages * (c.per + 32) <= SP_PART && c.per % 16 == 0, "stages %u per %u", c.stages, c.per);
                    u64 extent = c.rs ? c.rs * c.ndst : c.nu;
                    for (u64 row = row0; row < row1; row++) { u64 piece, q, r0; if (c.rs) { piece = row % pieces; q = row / pieces % c.nsrc; r0 = row / pieces / c.nsrc; } else { r0 = row % sets * c.group; piece = row / sets % pieces; q = row / sets / pieces; }
                        u64 p0 = piece * c.per, len = std::min<u64>(c.per, c.nu - p0), off = c.rs * r0 + p0, A = ps(q) + off, E = A + len;
                        u64 x0 = off >= 16 ? A & ~15ull : (A + 15) & ~15ull, x1 = off + len + 16 <= extent ? (E + 15) & ~15ull : E & ~15ull;
                        if (x1 > x0) { rd(q, x0, x1 - x0); CHK(x1 - x0 <= c.per + 32, "pitch"); }
                        u64 re = c.rs ? r0 + 1 : std::min<u64>(r0 + c.group, c.ndst);
                        for (u64 x = r0; x < re; x++) wr(pd(x), pd(x) + q * c.nu + p0, len); }
                } else CHK(0, "kind");
            }
        }
        for (int i = 0; i < P; i++) { long want = (long)(rl * es); if (op == 1 && i == d.root) want = 0; if (op == 2 && i != d.root) want = 0; CHK(wrote[rb[i].a] == want, "rank %d wrote %ld of %ld op %d P %d n %llu es %d", i, wrote[rb[i].a], want, op, P, n, es); }
    }
    printf("tiles %ld bad %ld kinds", tiles, bad); for (auto& k : kinds) printf(" %d:%ld", k.first, k.second); printf("\n");
    return bad != 0;
}
