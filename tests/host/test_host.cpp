// Host-side tests in the reference's own test style (one executable, local CHECK macro that
// prints and exits: tests/unit/test_kv_cache.cpp:10-17 of the reference).
//   test_host units            page table, planner and C++ wrapper checks that need no GPU
//   test_host rope f c th p..  prints cos/sin bits of the rotary table rows for positions p..
//   test_host decode in out    GPU: runs decode steps through the C++23 wrapper with host buffers
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <numeric>

#include "../../mugen_b200/csrc/mla_absorb_ring.h"
#include "../../mugen_b200/csrc/mla_few_ring.h"
#include "../../mugen_b200/host/mla_host.hpp"
#include "../../mugen_b200/host/page_table.hpp"
#include "../../mugen_b200/host/rope_table.hpp"
#include "../../mugen_b200/host/upload_order.hpp"

#define CHECK(cond)                                                              \
    do {                                                                         \
        if (!(cond)) {                                                           \
            std::fprintf(stderr, "CHECK failed %s:%d: %s\n", __FILE__, __LINE__, #cond); \
            std::exit(1);                                                        \
        }                                                                        \
    } while (0)

using namespace mugen::mla;

static void test_page_table()
{
    PageTable pt(64, 8, 3, 300);
    uint32_t a, b, c, d;
    CHECK(pt.seq_create(&a) == PT_OK && pt.seq_create(&b) == PT_OK && pt.seq_create(&c) == PT_OK);
    CHECK(pt.seq_create(&d) == PT_CAPACITY);
    CHECK(pt.reserve(a, 130) == PT_OK && pt.free_pages() == 5);     // 3 pages
    CHECK(pt.advance(a, 130) == PT_OK);
    CHECK(pt.advance(a, 63) == PT_INVALID);                         // beyond the reserved rows (192)
    CHECK(pt.reserve(b, 301) == PT_CAPACITY);                       // beyond max_seq_len
    CHECK(pt.reserve(b, 64 * 6) == PT_CAPACITY);
    CHECK(pt.reserve(b, 300) == PT_OK && pt.free_pages() == 0);     // 5 pages
    CHECK(pt.reserve(c, 1) == PT_NO_PAGES);
    uint32_t n = 0;
    CHECK(pt.seq_len(a, &n) == PT_OK && n == 130);
    CHECK(pt.truncate(a, 131) == PT_INVALID);                       // never grows
    CHECK(pt.truncate(a, 65) == PT_OK && pt.free_pages() == 1);     // keeps the partial page
    CHECK(pt.truncate(a, 64) == PT_OK && pt.free_pages() == 2);
    CHECK(pt.clear(a) == PT_OK && pt.free_pages() == 3);
    CHECK(pt.seq_len(a, &n) == PT_OK && n == 0);
    CHECK(pt.set_base(b, 10) == PT_INVALID);                        // only on an empty sequence
    CHECK(pt.set_base(a, 4096) == PT_OK);
    CHECK(pt.seq_free(b) == PT_OK && pt.free_pages() == 8);
    CHECK(pt.seq_len(b, &n) == PT_INVALID);
    // slots: distinct pages, offset within page
    CHECK(pt.reserve(c, 200) == PT_OK);
    CHECK(pt.slot(c, 0) % 64 == 0 && pt.slot(c, 63) == pt.slot(c, 0) + 63);
    CHECK(pt.slot(c, 64) / 64 != pt.slot(c, 0) / 64);
    // a shuffled free list still hands out every page exactly once
    PageTable p2(64, 100, 1, 6400);
    p2.shuffle_free(7);
    uint32_t s;
    CHECK(p2.seq_create(&s) == PT_OK && p2.reserve(s, 6400) == PT_OK);
    std::vector<int> seen(100, 0);
    for (uint32_t pg : p2.seq(s)->pages) seen[pg]++;
    for (int v : seen) CHECK(v == 1);
}

static void test_planner()
{
    std::vector<Segment> segs;
    std::vector<uint32_t> rsb, wsb;
    // uniform batch: equal shares, every page covered exactly once, in order
    std::vector<uint32_t> lens(64, 16384);
    plan_balanced(lens, 64, 74, segs, rsb, wsb);
    CHECK(wsb.size() == 75 && rsb.size() == 65);
    uint64_t covered = 0;
    for (uint32_t r = 0; r < 64; r++) {
        uint32_t next = 0;
        for (uint32_t g = rsb[r]; g < rsb[r + 1]; g++) {
            CHECK(segs[g].row == r && segs[g].page_begin == next && segs[g].page_end > next);
            next = segs[g].page_end;
        }
        CHECK(next == 256);
        covered += next;
    }
    CHECK(covered == 64 * 256);
    for (uint32_t w = 0; w < 74; w++) {
        uint64_t pages = 0;
        for (uint32_t g = wsb[w]; g < wsb[w + 1]; g++) pages += segs[g].page_end - segs[g].page_begin;
        CHECK(pages == 221 || pages == 222);
    }
    // ragged batch with empty rows; fewer pages than workers
    lens = {0, 1, 64, 65, 0, 1000, 0};
    plan_balanced(lens, 64, 148, segs, rsb, wsb);
    CHECK(rsb[1] - rsb[0] == 1 && segs[rsb[0]].page_begin == segs[rsb[0]].page_end);   // empty row keeps a segment
    uint64_t total = 0;
    for (auto& g : segs) total += g.page_end - g.page_begin;
    CHECK(total == 0 + 1 + 1 + 2 + 0 + 16 + 0);
    CHECK(wsb.back() == segs.size());
    for (size_t w = 0; w + 1 < wsb.size(); w++) CHECK(wsb[w] <= wsb[w + 1]);
    // one long row over many workers: one segment per worker
    lens = {131072};
    plan_balanced(lens, 64, 148, segs, rsb, wsb);
    CHECK(segs.size() == 148 && rsb[1] == 148);
    // two-page tiles: every cut inside a row falls on an even page, pages are still covered once, shares are
    // equal in tiles; a row with an odd page count keeps its last single page
    lens.assign(64, 16385);                                   // 257 pages = 129 tiles per row
    plan_balanced(lens, 64, 74, segs, rsb, wsb, 2);
    for (uint32_t r = 0; r < 64; r++) {
        uint32_t next = 0;
        for (uint32_t g = rsb[r]; g < rsb[r + 1]; g++) {
            CHECK(segs[g].row == r && segs[g].page_begin == next && segs[g].page_end > next);
            CHECK(segs[g].page_begin % 2 == 0);
            CHECK(segs[g].page_end % 2 == 0 || segs[g].page_end == 257);
            next = segs[g].page_end;
        }
        CHECK(next == 257);
    }
    for (uint32_t w = 0; w < 74; w++) {
        uint64_t tiles = 0;
        for (uint32_t g = wsb[w]; g < wsb[w + 1]; g++) tiles += (segs[g].page_end - segs[g].page_begin + 1) / 2;
        CHECK(tiles == 111 || tiles == 112);
    }
    lens = {0, 1, 64, 65, 0, 1000, 0};
    plan_balanced(lens, 64, 148, segs, rsb, wsb, 2);
    total = 0;
    for (auto& g : segs) total += g.page_end - g.page_begin;
    CHECK(total == 0 + 1 + 1 + 2 + 0 + 16 + 0);
    // nothing at all
    lens.clear();
    plan_balanced(lens, 64, 148, segs, rsb, wsb);
    CHECK(segs.empty() && rsb.size() == 1 && wsb.back() == 0);

    // ---- the plan that prices segments: coverage, order, cuts on tile boundaries, and a makespan no worse than
    // the equal-share plan's under the same price
    auto cost_of = [&](const std::vector<Segment>& sg, const std::vector<uint32_t>& ws, uint32_t ovh) {
        uint64_t worst = 0;
        for (size_t w = 0; w + 1 < ws.size(); w++) {
            uint64_t c = 0;
            for (uint32_t g = ws[w]; g < ws[w + 1]; g++) {
                const uint32_t n = sg[g].page_end - sg[g].page_begin;
                if (n) c += ovh + (n + 1) / 2;
            }
            worst = std::max(worst, c);
        }
        return worst;
    };
    for (auto cfg : std::vector<std::pair<std::vector<uint32_t>, uint32_t>>{
             {std::vector<uint32_t>(8, 16384), 74}, {std::vector<uint32_t>(64, 16384), 74}, {std::vector<uint32_t>(1, 131072), 74},
             {{0, 1, 64, 65, 0, 1000, 0, 32768, 300}, 74}, {std::vector<uint32_t>(3, 100), 148}, {{}, 74}}) {
        const auto& ls = cfg.first;
        std::vector<Segment> s2, s1;
        std::vector<uint32_t> r2, w2, r1, w1;
        plan_min_makespan(ls, 64, cfg.second, s2, r2, w2, 2, 4);
        CHECK(r2.size() == ls.size() + 1 && w2.back() == s2.size() && w2.size() <= cfg.second + 1u);
        for (uint32_t r = 0; r < ls.size(); r++) {
            uint32_t next = 0;
            CHECK(r2[r + 1] > r2[r]);                                   // every row keeps at least one segment
            for (uint32_t g = r2[r]; g < r2[r + 1]; g++) {
                CHECK(s2[g].row == r && s2[g].page_begin == next && s2[g].page_begin % 2 == 0);
                CHECK(s2[g].page_end > next || ls[r] == 0);
                next = s2[g].page_end;
            }
            CHECK(next == (ls[r] + 63) / 64);
        }
        for (size_t w = 0; w + 1 < w2.size(); w++) CHECK(w2[w] <= w2[w + 1]);
        if (!ls.empty()) {
            plan_balanced(ls, 64, cfg.second, s1, r1, w1, 2);
            CHECK(cost_of(s2, w2, 4) <= cost_of(s1, w1, 4));
        }
    }
    // the bounds of the search hold the answer: never more workers than there are, and one unit less would need more
    uint32_t rnd = 7;
    auto next_rnd = [&](uint32_t n) { rnd = rnd * 1664525u + 1013904223u; return (rnd >> 8) % n; };
    for (int rep = 0; rep < 2000; rep++) {
        std::vector<uint32_t> ls(1 + next_rnd(60));
        const uint32_t top = 1u << (1 + next_rnd(17)), workers = 1 + next_rnd(200), granule = 1 + next_rnd(2), price = next_rnd(5);
        for (auto& l : ls) l = next_rnd(4) ? next_rnd(top) : top;
        std::vector<Segment> s2;
        std::vector<uint32_t> r2, w2;
        plan_min_makespan(ls, 64, workers, s2, r2, w2, granule, price);
        CHECK(w2.size() <= workers + 1u);
        uint64_t worst = 0, work = 0;
        for (size_t w = 0; w + 1 < w2.size(); w++) {
            uint64_t load = 0;
            for (uint32_t g = w2[w]; g < w2[w + 1]; g++)
                if (const uint32_t n = s2[g].page_end - s2[g].page_begin) load += price + (n + granule - 1) / granule;
            worst = std::max(worst, load);
            work += load;
        }
        CHECK(worst * std::min<uint64_t>(workers, std::max<uint64_t>(work, 1)) >= work);
        CHECK(worst <= (work + (workers - 1)) / workers + 2 * price + 2);                // greedy: every worker but the last is full
    }
    {   // 8 rows of 128 tiles over 74 workers: nobody gets two segments for the price of one
        std::vector<Segment> s2;
        std::vector<uint32_t> r2, w2;
        plan_min_makespan(std::vector<uint32_t>(8, 16384), 64, 74, s2, r2, w2, 2, 4);
        CHECK(cost_of(s2, w2, 4) <= 19);
    }
}

// The absorb kernel's weight ring with its barriers as the hardware tests them: one bit of the phase number.  Copies in flight
// land in any order, an issuer may run one row tile ahead of the slowest (two query buffers), and a stage's release may lag.
// Random schedules; returns false where an issuer reads a piece that has not landed, a piece is requested into a stage that
// is still read, or nothing can move any more.
template <typename Stage, typename Parity>
static bool ring_holds(uint32_t n_d, uint32_t n_stages, uint32_t units, uint32_t seed, Stage stage, Parity parity)
{
    const auto passes = [](uint32_t completed, uint32_t bit) { return (completed & 1) != bit; };       // mbarrier.try_wait.parity
    std::vector<uint32_t> full(n_stages, 0), empty(n_stages, 0);          // completed phases
    std::vector<int> in(n_stages, -1);                                    // landed and not yet released piece of a stage
    std::vector<uint32_t> flying, released, at(n_d, 0), done(units, 0);   // at: an issuer's next piece; done: issuers past a unit
    const uint32_t pieces = units * 2 * n_d;
    uint32_t requested = 0, finished = 0;
    const auto where = [&](uint32_t p) { return stage((p / 2) % n_d, p / (2 * n_d), p % 2); };
    const auto bit = [&](uint32_t p) { return parity((p / 2) % n_d, p / (2 * n_d), p % 2); };
    while (finished < n_d || !released.empty()) {
        bool moved = false;
        for (uint32_t tries = 0; tries < 64 && !moved; tries++) {
            seed = seed * 1664525u + 1013904223u;
            const uint32_t pick = seed >> 16, act = pick % (n_d + 3);
            if (act == 0 && requested < pieces && passes(empty[where(requested)], bit(requested) ^ 1)) {
                const uint32_t s = where(requested);
                for (uint32_t f : flying) if (where(f) == s) return false;
                if (in[s] >= 0) return false;
                flying.push_back(requested++);
                moved = true;
            } else if (act == 1 && !flying.empty()) {
                const uint32_t k = (pick >> 4) % flying.size(), p = flying[k];
                flying.erase(flying.begin() + k);
                in[where(p)] = int(p);
                full[where(p)]++;
                moved = true;
            } else if (act == 2 && !released.empty()) {
                const uint32_t k = (pick >> 4) % released.size(), s = released[k];
                released.erase(released.begin() + k);
                in[s] = -1;
                empty[s]++;
                moved = true;
            } else if (act >= 3) {
                const uint32_t d = act - 3, unit = at[d] / 2;
                if (unit >= units || (unit >= 2 && done[unit - 2] < n_d)) continue;
                const uint32_t p = (unit * n_d + d) * 2 + at[d] % 2, s = where(p);
                if (!passes(full[s], bit(p))) continue;
                if (in[s] != int(p)) return false;
                released.push_back(s);
                at[d]++;
                if (at[d] % 2 == 0) done[unit]++;
                if (at[d] == 2 * units) finished++;
                moved = true;
            }
        }
        if (!moved) return false;
    }
    return true;
}

static void test_absorb_ring()
{
    for (uint32_t n_d : {1u, 2u, 4u})
        for (uint32_t per : {2u, 3u})
            for (uint32_t seed = 1; seed <= 300; seed++) {
                const mla::AbsorbRing ring{per};
                CHECK(ring_holds(n_d, 4 * per, 12, seed, [&](uint32_t d, uint32_t u, uint32_t h) { return ring.stage(d, u, h); },
                                 [&](uint32_t, uint32_t u, uint32_t h) { return ring.parity(u, h); }));
            }
    // a ring that all issuers share does not hold: the model finds the read ahead of the copy
    for (uint32_t stages : {10u, 12u}) {
        uint32_t broken = 0;
        for (uint32_t seed = 1; seed <= 300; seed++)
            broken += !ring_holds(4, stages, 12, seed, [&](uint32_t d, uint32_t u, uint32_t h) { return (8 * u + 2 * d + h) % stages; },
                                  [&](uint32_t d, uint32_t u, uint32_t h) { return ((8 * u + 2 * d + h) / stages) & 1; });
        CHECK(broken > 0);
    }
}

// The same for the few-row projection kernel: one block of kbs k-blocks, requested in order, landing in any; an issuer walks
// k-blocks p, next(p), .. on its own, and nothing holds it back but the stages' barriers.
template <typename Next>
static bool few_ring_holds(uint32_t kbs, uint32_t seed, Next next)
{
    using R = mla::FewRing;
    const auto passes = [](uint32_t completed, uint32_t bit) { return (completed & 1) != bit; };
    std::vector<uint32_t> full(R::stages, 0), empty(R::stages, 0), flying, released, at(R::issuers), seen(kbs, 0);
    std::vector<int> in(R::stages, -1);
    for (uint32_t p = 0; p < R::issuers; p++) at[p] = p;
    uint32_t requested = 0, left = kbs;
    while (left || !released.empty()) {
        bool moved = false;
        for (uint32_t tries = 0; tries < 128 && !moved; tries++) {
            seed = seed * 1664525u + 1013904223u;
            const uint32_t pick = seed >> 16, act = pick % (R::issuers + 3);
            if (act == 0 && requested < kbs && passes(empty[R::stage(requested)], R::parity(requested) ^ 1)) {
                const uint32_t s = R::stage(requested);
                for (uint32_t f : flying) if (R::stage(f) == s) return false;
                if (in[s] >= 0) return false;
                flying.push_back(requested++);
                moved = true;
            } else if (act == 1 && !flying.empty()) {
                const uint32_t k = (pick >> 4) % flying.size(), i = flying[k];
                flying.erase(flying.begin() + k);
                in[R::stage(i)] = int(i);
                full[R::stage(i)]++;
                moved = true;
            } else if (act == 2 && !released.empty()) {
                const uint32_t k = (pick >> 4) % released.size(), s = released[k];
                released.erase(released.begin() + k);
                in[s] = -1;
                empty[s]++;
                moved = true;
            } else if (act >= 3) {
                const uint32_t p = act - 3, i = at[p], s = R::stage(i);
                if (i >= kbs || !passes(full[s], R::parity(i))) continue;
                if (in[s] != int(i) || seen[i]++) return false;
                released.push_back(s);
                at[p] = next(i);
                left--;
                moved = true;
            }
        }
        if (!moved) return false;
    }
    return flying.empty();
}

static void test_few_ring()
{
    using R = mla::FewRing;
    for (uint32_t kbs = 1; kbs <= 32; kbs++)
        for (uint32_t seed = 1; seed <= 200; seed++) CHECK(few_ring_holds(kbs, seed, R::next));
    for (uint32_t i = 0; i < 64; i++) CHECK(R::issuer(R::next(i)) == R::issuer(i) && (i >= R::issuers || R::issuer(i) == i));
    // k-blocks dealt out in turn hold while no stage comes round again, and do not behind that
    const auto in_turn = [](uint32_t i) { return i + R::issuers; };
    uint32_t broken[17] = {};
    for (uint32_t kbs = 1; kbs <= 16; kbs++)
        for (uint32_t seed = 1; seed <= 3000; seed++) broken[kbs] += !few_ring_holds(kbs, seed, in_turn);
    for (uint32_t kbs = 1; kbs <= 16; kbs++) CHECK((broken[kbs] > 0) == (kbs > R::stages));
}

// Uploads and launches in any order on three streams.  A launch must wait for an upload that stands between it and the kernel before
// it on its stream, unless the region has been written anew since; no other launch needs to.  Returns (launches that did not wait and had to,
// launches that waited for nothing).
struct LastUpload {          // one upload remembered for all streams
    uint64_t stream = 0;
    bool fresh = false;
    void uploaded(size_t, uint64_t s) { stream = s; fresh = true; }
    bool open(uint64_t s) const { return fresh && stream == s; }
    void followed(uint64_t s) { if (stream == s) fresh = false; }
};
template <typename Order>
static std::pair<uint32_t, uint32_t> wrong_launches(uint32_t seed)
{
    Order order;
    uint32_t early = 0, late = 0, version = 0, latest[4] = {};
    std::vector<std::pair<uint32_t, uint32_t>> behind[3];       // (region, version) uploaded behind the last kernel of a stream
    for (int i = 0; i < 400; i++) {
        seed = seed * 1664525u + 1013904223u;
        const uint32_t s = (seed >> 8) % 3, r = (seed >> 16) % 4;
        if ((seed >> 24) % 2) {
            order.uploaded(r, 10 + s);
            latest[r] = ++version;
            behind[s].push_back({r, version});
        } else {
            bool must = false;
            for (auto [region, v] : behind[s]) must = must || latest[region] == v;
            early += must && !order.open(10 + s);
            late += !must && order.open(10 + s);
            order.followed(10 + s);
            behind[s].clear();
        }
    }
    return {early, late};
}

static void test_upload_order()
{
    UploadOrder<4> order;
    CHECK(!order.open(0));                                   // 0 is a stream like any other
    order.uploaded(0, 7);                                    // step_begin on one stream, a group of layers on another
    order.uploaded(2, 8);
    CHECK(order.open(7) && order.open(8) && !order.open(9));
    order.followed(8);
    CHECK(order.open(7) && !order.open(8));
    order.uploaded(0, 8);                                    // the next step, on the other stream
    CHECK(!order.open(7) && order.open(8));
    order.followed(8);
    CHECK(!order.open(7) && !order.open(8));
    uint32_t early = 0;
    for (uint32_t seed = 1; seed <= 500; seed++) {
        CHECK(wrong_launches<UploadOrder<4>>(seed) == std::make_pair(0u, 0u));
        early += wrong_launches<LastUpload>(seed).first;
    }
    CHECK(early > 0);
}

static void test_wrapper_without_gpu()
{
    LatentKVCacheConfig cfg;
    cfg.n_layers = 0;
    auto bad = LatentKVCache::create(cfg);
    CHECK(!bad && bad.error() == "n_layers must be > 0");    // KVCache::create's message
}

static std::vector<char> slurp(const char* path)
{
    std::ifstream f(path, std::ios::binary);
    return std::vector<char>((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
}

// Input file: u32 header {H, L, B, T, bf16} then weights per layer (w_uk, w_uv as 16-bit values,
// norm[512]) then per step per layer kv_a[B][576], q[B][H][192].  Output: out[T][L][B][H][128].
static int run_decode(const char* in_path, const char* out_path)
{
    auto buf = slurp(in_path);
    const auto* hdr = reinterpret_cast<const uint32_t*>(buf.data());
    const uint32_t H = hdr[0], L = hdr[1], B = hdr[2], T = hdr[3], bf16 = hdr[4];
    const uint16_t* p = reinterpret_cast<const uint16_t*>(buf.data() + 20);
    LatentKVCacheConfig cfg;
    cfg.n_layers = L; cfg.n_heads = H; cfg.max_seq_len = 256; cfg.n_pages = 4 * B; cfg.max_seqs = B;
    cfg.bf16 = bf16 != 0; cfg.rope_scaling_factor = 40.0f; cfg.rope_original_ctx = 4096; cfg.rms_norm_eps = 1e-6f;
    auto cache = LatentKVCache::create(cfg);
    if (!cache) { std::fprintf(stderr, "create: %s\n", cache.error().c_str()); return 2; }
    MlaAttention attn(**cache);
    const size_t wn = size_t(H) * 128 * 512;
    for (uint32_t l = 0; l < L; l++) {
        auto r = attn.set_layer_weights(l, p, p + wn, bf16 ? MLA_W_BF16 : MLA_W_F16, p + 2 * wn);
        if (!r) { std::fprintf(stderr, "weights: %s\n", r.error().c_str()); return 2; }
        p += 2 * wn + 512;
    }
    std::vector<uint32_t> seqs(B);
    for (auto& s : seqs) s = (*cache)->new_sequence().value();
    std::vector<uint16_t> out(size_t(T) * L * B * H * 128);
    uint16_t* o = out.data();
    for (uint32_t t = 0; t < T; t++) {
        if (auto r = attn.step_begin(seqs); !r) { std::fprintf(stderr, "begin: %s\n", r.error().c_str()); return 2; }
        for (uint32_t l = 0; l < L; l++) {
            const uint16_t* kv = p;
            const uint16_t* q = p + size_t(B) * 576;
            p += size_t(B) * 576 + size_t(B) * H * 192;
            if (auto r = attn.step_layer_host(l, kv, q, o); !r) { std::fprintf(stderr, "layer: %s\n", r.error().c_str()); return 2; }
            o += size_t(B) * H * 128;
        }
        if (auto r = attn.step_end(); !r) return 2;
        CHECK((*cache)->seq_len(seqs[0]) == t + 1);
    }
    if (auto r = attn.check_device(); !r) { std::fprintf(stderr, "device: %s\n", r.error().c_str()); return 2; }
    CHECK((*cache)->truncate(seqs[0], T + 1).has_value() == false);
    std::ofstream f(out_path, std::ios::binary);
    f.write(reinterpret_cast<const char*>(out.data()), out.size() * 2);
    return 0;
}

int main(int argc, char** argv)
{
    if (argc >= 2 && !std::strcmp(argv[1], "units")) {
        test_page_table();
        test_planner();
        test_absorb_ring();
        test_few_ring();
        test_upload_order();
        test_wrapper_without_gpu();
        std::puts("host units ok");
        return 0;
    }
    if (argc >= 6 && !std::strcmp(argv[1], "rope")) {
        const float factor = std::strtof(argv[2], nullptr);
        const uint32_t ctx = uint32_t(std::strtoul(argv[3], nullptr, 10));
        const float theta = std::strtof(argv[4], nullptr);
        for (int i = 5; i < argc; i++) {
            const uint32_t pos = uint32_t(std::strtoul(argv[i], nullptr, 10));
            float row[64];
            fill_rope_rows(row, pos, pos + 1, factor, ctx, theta);
            for (int k = 0; k < 64; k++) {
                uint32_t u;
                std::memcpy(&u, &row[k], 4);
                std::printf("%08x%c", u, k == 63 ? '\n' : ' ');
            }
        }
        return 0;
    }
    if (argc >= 4 && !std::strcmp(argv[1], "decode")) return run_decode(argv[2], argv[3]);
    std::fprintf(stderr, "usage: test_host units | rope factor ctx theta pos... | decode in out\n");
    return 64;
}
