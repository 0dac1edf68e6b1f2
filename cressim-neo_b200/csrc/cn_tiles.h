// cn_tiles.h -- host side of the tiled soft iteration: cuts a scene's particles into compact tiles
// and each constraint family into the entries every tile has to solve.
//
// A tile owns some particles and lists every constraint that touches one of them, so one CTA can
// solve a family on its particles without leaving the SM: it reads the positions of its own and
// its halo particles, solves its entries, sums each own particle's corrections in ascending
// constraint order (the order of the per-family gather) and writes the new positions.  A
// constraint across tiles is solved by each of them, to the same bits.
#pragma once

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <memory>
#include <new>
#include <thread>
#include <utility>
#include <vector>

#include "cn_device.h"
#include "cn_internal.h"

namespace cn {

constexpr uint32_t kTileSmemCap = 112u << 10; // two tiles' CTAs on an SM
// Particles per tile for the n particles of a world that go into tiles, whatever else is in it; 0: the
// per-family kernels run.
//  * A small scene is all latency, and a CTA's threads should each have one entry or two of a stage: tiles
//    of 16 (lattices of 216 to 2,744 particles, 4 substeps x 20 iterations, per frame: 547-612 us with the
//    per-family kernels, 400-460 us with tiles of 12 to 24, 410-515 us with tiles of 48).
//  * Large scenes fill whole waves of two CTAs an SM with tiles of at most 192 (a larger tile solves
//    fewer constraints twice, but 340 leaves too few CTAs: 100K particles, 4 x 20 iterations, 2.4 ms at
//    170, 2.9 at 96, 2.7 at 340, 4.0 with the per-family kernels).  16K of tissue and cloth, 2 x 20 iterations:
//    1,217 us with the per-family kernels, 1,140 with tiles of 55, 1,206 of 64, 1,403 of 16.
//  * Beside a fluid that fills the chip (`fluid`) work done twice is the fluid's time: no tiles from 1,536 to
//    24,576 particles, of at least 144 above.  7K of tissue and cloth beside 50K of fluid, 2 x 20 iterations:
//    3,555 us with the per-family kernels, 4,000 with tiles of 32, 3,610 of 96, 3,555 of 144; 17K beside 64K, 2 x 8:
//    2,170, of 59 2,285, of 144 2,210; 38K beside 157K, 1 x 20: 2,600, of 129 2,585, of 144 2,580; 60K beside 130K,
//    2 x 10: 7,754, of 144 7,690; 1K beside 130K, 2 x 20 (2 of the fluid): 2,267, of 16 2,130.
//  * In between the per-family kernels stay, though the tiles measured faster there as well (4,096
//    particles: 505 against 647 us): the frame graph of the 16^3 cube is held to one launch per
//    phase by the schedule test, which the stages' two launches an iteration do not meet.
inline uint32_t tileTarget(uint32_t n, bool fluid)
{
    if (n <= (fluid ? 1536u : 3072u)) return 16u;
    if (n < (fluid ? 24576u : 6144u)) return 0u;
    constexpr uint32_t kWave = 2u * 148u;
    uint32_t waves = 1u;
    while (n > kWave * waves * 192u) ++waves;
    return std::max((n + kWave * waves - 1u) / (kWave * waves), fluid ? 144u : 32u);
}

// A vector whose new elements are left as they are: the lists are written, not zeroed first.
template <class T> struct TileAllocator : std::allocator<T> {
    template <class U> struct rebind {
        using other = TileAllocator<U>;
    };
    template <class U> void construct(U *p) noexcept { ::new (static_cast<void *>(p)) U; }
    template <class U, class... A> void construct(U *p, A &&...a) { ::new (static_cast<void *>(p)) U(std::forward<A>(a)...); }
};
template <class T> using TileVector = std::vector<T, TileAllocator<T>>;

struct TileBuild {
    bool ok = false;
    TileVector<TileHead> heads;
    TileVector<uint32_t> own, halo;
    TileVector<uint32_t> rec[2];       // per own particle (tileRecord)
    TileVector<uint32_t> id[2];        // per entry: constraint
    TileVector<uint2> edges;           // stage 0 entries (TileSet::edges)
    TileVector<uint4> elems;           // stage 1 entries (TileSet::elems)
    uint32_t smem[2] = {0, 0};         // dynamic shared memory of the largest tile, per stage
};

// What the builder reads of a scene.  Class 0 particles are left out, class 1 particles have tets (or
// no second family), class 2 particles have bends / dihedrals; a tile holds one class.
template <class EdgeOf, class TetOf, class BendOf> struct TileInput {
    uint32_t n;
    const float *positions;            // float4[n]
    const std::vector<uint8_t> &cls;
    const Incidence &edgeI, &tetI, &bendI;
    EdgeOf edgeOf;
    TetOf tetOf;
    BendOf bendOf;
};

// A particle of the bisection: its coordinates as keys that order like them (zero where not finite) beside
// its index, so that a cut runs over contiguous memory.
struct TileParticle {
    uint32_t at[3];
    uint32_t id;
};
inline uint32_t tileKey(float v)
{
    if (!std::isfinite(v)) v = 0.0f;
    v += 0.0f; // one zero
    uint32_t u;
    std::memcpy(&u, &v, 4);
    return u >> 31 ? ~u : u | 0x80000000u;
}
inline float tileCoordinate(uint32_t key)
{
    const uint32_t u = key >> 31 ? key & 0x7fffffffu : ~key;
    float v;
    std::memcpy(&v, &u, 4);
    return v;
}

// Cuts parts[b, e) across its longest side into left : tiles - left; returns the cut.  The particles are in
// the order of their indices and stay so on both sides; of equal coordinates the lower indices go left.  A
// selection by digits of the key: std::nth_element meets its worst case on lattices.  `buffer`: scratch of
// e entries.
inline uint32_t tileCut(std::vector<TileParticle> &parts, std::vector<TileParticle> &buffer, uint32_t b, uint32_t e, uint32_t left,
                        uint32_t tiles)
{
    uint32_t lo[3], hi[3];
    for (int a = 0; a < 3; ++a) lo[a] = hi[a] = parts[b].at[a];
    for (uint32_t i = b + 1; i < e; ++i)
        for (int a = 0; a < 3; ++a) {
            lo[a] = std::min(lo[a], parts[i].at[a]);
            hi[a] = std::max(hi[a], parts[i].at[a]);
        }
    int axis = 0;
    float most = -1.0f;
    for (int a = 0; a < 3; ++a) {
        const float side = tileCoordinate(hi[a]) - tileCoordinate(lo[a]);
        if (side > most) {
            most = side;
            axis = a;
        }
    }
    uint32_t mid = b + uint32_t(uint64_t(e - b) * left / tiles);
    mid = std::min(std::max(mid, b + 1u), e - 1u);
    // the key of rank `mid`, a digit at a time (few digits for few particles), and how many of its equals go left
    const uint32_t width = e - b < 4096u ? 8u : 11u;
    uint32_t key = 0, mask = 0, rank = mid - b;
    for (uint32_t high = 32u; high > 0u;) {
        const uint32_t shift = high > width ? high - width : 0u, digits = (1u << (high - shift)) - 1u;
        std::array<uint32_t, 2048> count;
        std::fill(count.begin(), count.begin() + digits + 1u, 0u);
        for (uint32_t i = b; i < e; ++i) {
            const uint32_t k = parts[i].at[axis];
            if ((k & mask) == key) ++count[(k >> shift) & digits];
        }
        uint32_t digit = 0;
        while (rank >= count[digit]) rank -= count[digit++];
        key |= digit << shift;
        mask |= digits << shift;
        high = shift;
    }
    uint32_t to = b, kept = 0;
    for (uint32_t i = b; i < e; ++i) {
        const uint32_t k = parts[i].at[axis];
        if (k < key || (k == key && rank > 0u && rank--)) parts[to++] = parts[i];
        else buffer[b + kept++] = parts[i];
    }
    std::copy(buffer.begin() + b, buffer.begin() + b + kept, parts.begin() + to);
    return mid;
}

// The local indices of a tile's particles: a word per particle of the scene, stamped with the tile.  The
// words come zeroed from the system, which backs the pages that are used: those of a worker's own tiles.
class TileLocals {
public:
    explicit TileLocals(uint32_t n) : words(static_cast<uint64_t *>(std::calloc(std::max(n, 1u), sizeof(uint64_t))), &std::free)
    {
        if (!words) throw std::bad_alloc();
    }
    void next() { ++stamp; }
    static constexpr uint32_t kNone = 0xffffffffu;
    uint32_t get(uint32_t x) const
    {
        const uint64_t w = words.get()[x];
        return uint32_t(w >> 32) == stamp ? uint32_t(w) : kNone;
    }
    void set(uint32_t x, uint32_t local) { words.get()[x] = uint64_t(stamp) << 32 | local; }

private:
    std::unique_ptr<uint64_t, void (*)(void *)> words;
    uint32_t stamp = 0;
};

// Builds the tiles of some leaves of the bisection, whose lists (TileBuild) buildTiles puts together in the
// leaves' order.  What it holds beside them is of the size of a tile (and the words of TileLocals), so that a
// large scene's memory does not multiply by its workers.
template <class In> class TileBuilder {
public:
    TileBuilder(const In &input, std::vector<TileParticle> &particles, std::vector<TileParticle> &scratch, size_t smemCap)
        : in(input), parts(particles), buffer(scratch), cap(smemCap), locals(input.n)
    {
        out.ok = true;
    }

    // The tiles of particles [b, e): one, or the halves of one over a limit.
    void leaf(uint32_t b, uint32_t e, bool bends)
    {
        if (!out.ok || b >= e || emit(b, e, bends)) return;
        if (e - b <= 1u) {
            out.ok = false;
            return;
        }
        std::sort(parts.begin() + b, parts.begin() + e, [](const TileParticle &x, const TileParticle &y) { return x.id < y.id; });
        const uint32_t mid = tileCut(parts, buffer, b, e, 1u, 2u);
        leaf(b, mid, bends);
        leaf(mid, e, bends);
    }

    TileBuild out;

private:
    struct Entry {
        uint32_t constraint;
        uint32_t local[4], slot[4];
    };
    // Entries of like shape (the same steps between their local indices) side by side, ascending in the first
    // particle: on a lattice a warp's threads then read neighbouring positions and write neighbouring record
    // slots, free of bank conflicts.  By counting, from the last key to the first (a comparison sort's
    // mispredicted branches took most of the lists' time).
    void sortEntries(int f, uint32_t particles)
    {
        const std::vector<Entry> &en = entries[f];
        const uint32_t n = uint32_t(en.size());
        std::vector<uint32_t> &to = sorted[f];
        to.resize(n);
        passed.resize(n);
        keys.resize(n);
        for (uint32_t i = 0; i < n; ++i) to[i] = i;
        for (uint32_t key : {0u, 3u, 2u, 1u}) {
            if (f == 0 && key > 1u) continue; // an edge has one step
            starts.assign(2u * particles + 1u, 0u);
            for (uint32_t i = 0; i < n; ++i) {
                // a step in 16 bits, its negative values after the others, as a number below 2 * particles
                const uint32_t *l = en[to[i]].local, base = key ? l[0] : 0u;
                keys[i] = l[key] - base + (2u * particles & (0u - uint32_t(l[key] < base)));
                ++starts[keys[i] + 1u];
            }
            for (uint32_t i = 0; i < 2u * particles; ++i) starts[i + 1u] += starts[i];
            for (uint32_t i = 0; i < n; ++i) passed[starts[keys[i]]++] = to[i];
            passed.swap(to);
        }
    }
    // Where an own particle's records of a family begin: in its incidence list, and their slots.
    struct Records {
        uint32_t first, base, width;
    };

    // The entries of a family, each where its first own particle lists it, and the particles around.
    template <uint32_t kPer, class Elem> void collect(const Incidence &inc, Elem &&elem, uint32_t b, uint32_t p, int f)
    {
        records.resize(p);
        for (uint32_t i = 0; i < p; ++i)
            records[i] = Records{inc.ranges[parts[b + i].id].x, tileRecordBase(rec[f][i]), tileRecordWidth(rec[f][i])};
        entries[f].clear();
        for (uint32_t i = 0; i < p; ++i) {
            const uint2 r = inc.ranges[parts[b + i].id];
            for (uint32_t q = r.x; q < r.x + r.y; ++q) {
                const uint32_t c = inc.inc[q].x, at = inc.inc[q].y;
                uint32_t x[kPer], l[kPer];
                bool listed = false; // without branches: half of them are
                for (uint32_t k = 0; k < kPer; ++k) {
                    x[k] = elem(c, k);
                    l[k] = x[k] < in.n ? locals.get(x[k]) : TileLocals::kNone;
                    listed |= (l[k] < i) | ((l[k] == i) & (k < at));
                }
                if (listed) continue;
                Entry &en = entries[f].emplace_back();
                en.constraint = c;
                for (uint32_t k = 0; k < 4u; ++k) {
                    en.local[k] = 0u;
                    en.slot[k] = kTileNoSlot;
                    if (k >= kPer || x[k] >= in.n) continue;
                    if (l[k] == TileLocals::kNone) l[k] = locals.get(x[k]); // a halo particle may be named twice
                    if (l[k] == TileLocals::kNone) {
                        l[k] = p + uint32_t(halo.size());
                        locals.set(x[k], l[k]);
                        halo.push_back(x[k]);
                    }
                    en.local[k] = l[k];
                    if (l[k] < p)
                        en.slot[k] = records[l[k]].base + (inc.dst[size_t(c) * kPer + k] - records[l[k]].first) * records[l[k]].width;
                }
            }
        }
    }
    // Emits the tile of particles [b, e) of `parts`; false when it is over a limit.
    bool emit(uint32_t b, uint32_t e, bool bends)
    {
        const uint32_t p = e - b, per[2] = {2u, 4u};
        const Incidence *inc[2] = {&in.edgeI, bends ? &in.bendI : &in.tetI};
        // like degrees side by side: a warp's threads then sum about as many records each
        std::sort(parts.begin() + b, parts.begin() + e, [&](const TileParticle &x, const TileParticle &y) {
            const uint32_t tx = inc[1]->ranges[x.id].y, ty = inc[1]->ranges[y.id].y;
            if (tx != ty) return tx > ty;
            const uint32_t ex = inc[0]->ranges[x.id].y, ey = inc[0]->ranges[y.id].y;
            return ex != ey ? ex > ey : x.id < y.id;
        });
        locals.next();
        for (uint32_t i = 0; i < p; ++i) locals.set(parts[b + i].id, i);
        // record slots in slices of 32 particles (the last one narrower): record q of a slice's
        // particle j at base + q * width + j, so a warp's q-th records are adjacent
        uint32_t slots[2] = {0u, 0u};
        for (int f = 0; f < 2; ++f) {
            rec[f].resize(p);
            for (uint32_t s0 = 0; s0 < p; s0 += 32u) {
                const uint32_t width = std::min(32u, p - s0);
                uint32_t most = 0;
                for (uint32_t i = s0; i < s0 + width; ++i) {
                    const uint32_t cnt = inc[f]->ranges[parts[b + i].id].y;
                    if (cnt > kTileMaxRecords || slots[f] + width > 0xfffeu) return false;
                    most = std::max(most, cnt);
                    rec[f][i] = tileRecord(slots[f] + (i - s0), width, cnt);
                }
                slots[f] += most * width;
                if (slots[f] > 0xfffeu) return false;
            }
        }
        halo.clear();
        collect<2u>(in.edgeI, in.edgeOf, b, p, 0);
        if (bends) collect<4u>(in.bendI, in.bendOf, b, p, 1);
        else collect<4u>(in.tetI, in.tetOf, b, p, 1);
        const size_t pos = size_t(p) + halo.size();
        if (pos > 0xffffu) return false;
        size_t need[2];
        for (int f = 0; f < 2; ++f) {
            need[f] = pos * 16 + size_t(slots[f]) * 12;
            if (need[f] > cap) return false;
        }
        order = halo; // as first met: what its local index becomes
        std::sort(halo.begin(), halo.end());
        for (uint32_t k = 0; k < halo.size(); ++k) locals.set(halo[k], p + k);
        for (uint32_t &x : order) x = locals.get(x);
        for (int f = 0; f < 2; ++f) {
            for (Entry &en : entries[f])
                for (uint32_t k = 0; k < per[f]; ++k)
                    if (en.local[k] >= p) en.local[k] = order[en.local[k] - p];
            sortEntries(f, uint32_t(pos));
        }

        TileHead h{};
        h.own = uint32_t(out.own.size());
        h.ownCount = p;
        h.halo = uint32_t(out.halo.size());
        h.haloCount = uint32_t(halo.size());
        h.bends = bends ? 1u : 0u;
        for (int f = 0; f < 2; ++f) {
            h.entry[f] = uint32_t(out.id[f].size());
            h.entryCount[f] = uint32_t(entries[f].size());
            h.slots[f] = slots[f];
            out.smem[f] = std::max(out.smem[f], uint32_t(need[f]));
            out.rec[f].insert(out.rec[f].end(), rec[f].begin(), rec[f].end());
            for (uint32_t k : sorted[f]) {
                const uint32_t *l = entries[f][k].local, *s = entries[f][k].slot;
                out.id[f].push_back(entries[f][k].constraint);
                if (f == 0) out.edges.push_back(make_uint2(l[0] | (l[1] << 16), s[0] | (s[1] << 16)));
                else out.elems.push_back(make_uint4(l[0] | (l[1] << 16), l[2] | (l[3] << 16), s[0] | (s[1] << 16), s[2] | (s[3] << 16)));
            }
        }
        for (uint32_t i = b; i < e; ++i) out.own.push_back(parts[i].id);
        out.halo.insert(out.halo.end(), halo.begin(), halo.end());
        out.heads.push_back(h);
        return true;
    }

    const In &in;
    std::vector<TileParticle> &parts, &buffer;
    const size_t cap;
    TileLocals locals;
    std::vector<uint32_t> rec[2], halo, order, sorted[2];
    std::vector<Entry> entries[2];
    std::vector<Records> records;               // of collect
    std::vector<uint32_t> starts, passed, keys; // of sortEntries
};

// Runs f(0) .. f(n - 1), on threads of their own where there are several; an exception of any is passed on.
template <class F> void runParallel(uint32_t n, F &&f)
{
    std::vector<std::exception_ptr> errors(n);
    auto guarded = [&](uint32_t k) {
        try {
            f(k);
        } catch (...) {
            errors[k] = std::current_exception();
        }
    };
    std::vector<std::thread> threads;
    uint32_t started = 1;
    for (; started < n; ++started) {
        try {
            threads.emplace_back(guarded, started);
        } catch (const std::exception &) { // no thread to be had (or no room to hold it): the caller runs the rest
            break;
        }
    }
    guarded(0);
    for (uint32_t k = started; k < n; ++k) guarded(k);
    for (std::thread &t : threads) t.join();
    for (const std::exception_ptr &e : errors)
        if (e) std::rethrow_exception(e);
}

// `target` particles per tile; a tile whose shared memory would exceed `smemCap` is halved.
// ok = false when the scene does not fit the tile records (the per-family kernels run then).
template <class EdgeOf, class TetOf, class BendOf>
TileBuild buildTiles(const TileInput<EdgeOf, TetOf, BendOf> &in, uint32_t target, size_t smemCap)
{
    using In = TileInput<EdgeOf, TetOf, BendOf>;
    using Builder = TileBuilder<In>;
    struct Leaf {
        uint32_t begin, end;
    };
    TileBuild out;
    out.ok = true;
    for (uint8_t c = 1; c <= 2; ++c) {
        std::vector<TileParticle> parts;
        for (uint32_t i = 0; i < in.n; ++i) {
            if (in.cls[i] != c) continue;
            const float *x = in.positions + 4 * size_t(i);
            parts.push_back(TileParticle{{tileKey(x[0]), tileKey(x[1]), tileKey(x[2])}, i});
        }
        if (parts.empty()) continue;
        std::vector<TileParticle> buffer(parts.size());
        // recursive bisection into leaves of equal size, in depth-first order
        const uint32_t count = uint32_t(parts.size()), tiles = (count + target - 1u) / target;
        // the lists take ~1 us a particle on one thread: one for every 256 particles, up to 16
        const uint32_t workers = std::min({std::max(count / 256u, 1u), std::max(std::thread::hardware_concurrency(), 1u), 16u});
        auto split = [&](auto &&self, uint32_t b, uint32_t e, uint32_t t, uint32_t threads) -> std::vector<Leaf> {
            if (t <= 1u || e - b <= 1u) return {Leaf{b, e}};
            const uint32_t left = t / 2u, mid = tileCut(parts, buffer, b, e, left, t);
            std::vector<Leaf> half[2];
            runParallel(threads > 1u ? 2u : 1u, [&](uint32_t k) {
                if (k == 0u) half[0] = self(self, b, mid, left, threads / 2u);
                if (k == 1u || threads <= 1u) half[1] = self(self, mid, e, t - left, threads / 2u);
            });
            half[0].insert(half[0].end(), half[1].begin(), half[1].end());
            return std::move(half[0]);
        };
        const std::vector<Leaf> leaves = split(split, 0u, count, tiles, workers);
        const uint32_t shares = std::min<uint32_t>(workers, uint32_t(leaves.size()));
        std::vector<TileBuild> built(shares);
        runParallel(shares, [&](uint32_t k) {
            Builder b(in, parts, buffer, smemCap);
            for (size_t l = leaves.size() * k / shares; l < leaves.size() * (k + 1u) / shares; ++l)
                b.leaf(leaves[l].begin, leaves[l].end, c == 2);
            built[k] = std::move(b.out);
        });
        for (const TileBuild &t : built)
            if (!t.ok) return TileBuild{};
        // put together behind what is there, each share at its place
        auto gather = [&](auto list) {
            auto &to = list(out);
            std::vector<size_t> at(shares + 1u, to.size());
            for (uint32_t k = 0; k < shares; ++k) at[k + 1u] = at[k] + list(built[k]).size();
            to.resize(at[shares]);
            return at;
        };
        const auto heads = [](TileBuild &t) -> auto & { return t.heads; };
        const auto own = [](TileBuild &t) -> auto & { return t.own; };
        const auto halo = [](TileBuild &t) -> auto & { return t.halo; };
        const auto edges = [](TileBuild &t) -> auto & { return t.edges; };
        const auto elems = [](TileBuild &t) -> auto & { return t.elems; };
        const auto rec0 = [](TileBuild &t) -> auto & { return t.rec[0]; };
        const auto rec1 = [](TileBuild &t) -> auto & { return t.rec[1]; };
        const auto id0 = [](TileBuild &t) -> auto & { return t.id[0]; };
        const auto id1 = [](TileBuild &t) -> auto & { return t.id[1]; };
        const std::vector<size_t> headAt = gather(heads), ownAt = gather(own), haloAt = gather(halo), edgeAt = gather(edges),
                                  elemAt = gather(elems), idAt[2] = {gather(id0), gather(id1)};
        gather(rec0);
        gather(rec1);
        runParallel(shares, [&](uint32_t k) {
            TileBuild &t = built[k];
            for (TileHead &h : t.heads) {
                h.own += uint32_t(ownAt[k]);
                h.halo += uint32_t(haloAt[k]);
                for (int f = 0; f < 2; ++f) h.entry[f] += uint32_t(idAt[f][k]);
            }
            auto copy = [](auto &to, const auto &from, size_t at) { std::copy(from.begin(), from.end(), to.begin() + at); };
            copy(out.heads, t.heads, headAt[k]);
            copy(out.own, t.own, ownAt[k]);
            copy(out.halo, t.halo, haloAt[k]);
            copy(out.edges, t.edges, edgeAt[k]);
            copy(out.elems, t.elems, elemAt[k]);
            for (int f = 0; f < 2; ++f) {
                copy(out.rec[f], t.rec[f], ownAt[k]);
                copy(out.id[f], t.id[f], idAt[f][k]);
            }
        });
        for (const TileBuild &t : built)
            for (int f = 0; f < 2; ++f) out.smem[f] = std::max(out.smem[f], t.smem[f]);
    }
    out.ok = !out.heads.empty();
    return out;
}

} // namespace cn
