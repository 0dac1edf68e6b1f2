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
#include <cmath>
#include <cstdint>
#include <exception>
#include <thread>
#include <tuple>
#include <utility>
#include <vector>

#include "cn_device.h"
#include "cn_internal.h"

namespace cn {

constexpr uint32_t kTileSmemCap = 112u << 10; // two tiles' CTAs on an SM
// Particles per tile; 0: the per-family kernels run.
//  * A small scene is all latency, and a CTA's threads should each have one entry or two of a stage: tiles
//    of 16 (lattices of 216 to 2,744 particles, 4 substeps x 20 iterations, per frame: 547-612 us with the
//    per-family kernels, 400-460 us with tiles of 12 to 24, 410-515 us with tiles of 48).
//  * Large scenes fill whole waves of two CTAs an SM with tiles of at most 192 (a larger tile solves
//    fewer constraints twice, but 340 leaves too few CTAs: 100K particles, 4 x 20 iterations, 2.4 ms at
//    170, 2.9 at 96, 2.7 at 340, 4.0 with the per-family kernels).
//  * In between the per-family kernels stay, though the tiles measured faster there as well (4,096
//    particles: 505 against 647 us): the frame graph of the 16^3 cube is held to one launch per
//    phase by the schedule test, which the stages' two launches an iteration do not meet.
inline uint32_t tileTarget(uint32_t n)
{
    if (n <= 3072u) return 16u;
    if (n < 6144u) return 0u;
    constexpr uint32_t kWave = 2u * 148u;
    uint32_t waves = 1u;
    while (n > kWave * waves * 192u) ++waves;
    return std::max((n + kWave * waves - 1u) / (kWave * waves), 32u);
}

struct TileBuild {
    bool ok = false;
    std::vector<TileHead> heads;
    std::vector<uint32_t> own, halo;
    std::vector<uint32_t> rec[2];      // per own particle (tileRecord)
    std::vector<uint32_t> id[2];       // per entry: constraint
    std::vector<uint2> edges;          // stage 0 entries (TileSet::edges)
    std::vector<uint4> elems;          // stage 1 entries (TileSet::elems)
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

// Builds the tiles of some leaves of the bisection: the stamps a tile's lists are collected with, and the
// lists themselves (TileBuild), which buildTiles puts together in the leaves' order.
template <class In> class TileBuilder {
public:
    TileBuilder(const In &input, std::vector<uint32_t> &particles, size_t smemCap)
        : in(input), parts(particles), cap(smemCap), localOf(input.n, 0u), stamp(input.n, 0xffffffffu)
    {
        const size_t constraints[2] = {in.edgeI.dst.size() / 2, std::max(in.tetI.dst.size(), in.bendI.dst.size()) / 4};
        for (int f = 0; f < 2; ++f) {
            entryOf[f].assign(constraints[f], 0u);
            entryStamp[f].assign(constraints[f], 0xffffffffu);
        }
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
        const uint32_t mid = bisect(in, parts, b, e, 1u, 2u);
        leaf(b, mid, bends);
        leaf(mid, e, bends);
    }

    // Cuts parts[b, e) across its longest side into left : tiles - left; returns the cut.
    static uint32_t bisect(const In &in, std::vector<uint32_t> &parts, uint32_t b, uint32_t e, uint32_t left, uint32_t tiles)
    {
        auto coord = [&](uint32_t p, int a) {
            const float c = in.positions[4 * size_t(p) + a];
            return std::isfinite(c) ? c : 0.0f;
        };
        int axis = 0;
        float most = -1.0f;
        for (int a = 0; a < 3; ++a) {
            float lo = coord(parts[b], a), hi = lo;
            for (uint32_t i = b + 1; i < e; ++i) {
                const float c = coord(parts[i], a);
                lo = std::min(lo, c);
                hi = std::max(hi, c);
            }
            if (hi - lo > most) {
                most = hi - lo;
                axis = a;
            }
        }
        uint32_t mid = b + uint32_t(uint64_t(e - b) * left / tiles);
        mid = std::min(std::max(mid, b + 1u), e - 1u);
        std::nth_element(parts.begin() + b, parts.begin() + mid, parts.begin() + e, [&](uint32_t x, uint32_t y) {
            const float cx = coord(x, axis), cy = coord(y, axis);
            return cx != cy ? cx < cy : x < y;
        });
        return mid;
    }

    TileBuild out;

private:
    // Emits the tile of particles [b, e) of `parts`; false when it is over a limit.
    bool emit(uint32_t b, uint32_t e, bool bends)
    {
        const uint32_t p = e - b, n = in.n, mark = attempt++;
        const Incidence *inc[2] = {&in.edgeI, bends ? &in.bendI : &in.tetI};
        const uint32_t per[2] = {2u, 4u};
        auto elem = [&](int f, uint32_t c, uint32_t k) -> uint32_t {
            return f == 0 ? in.edgeOf(c, k) : (bends ? in.bendOf(c, k) : in.tetOf(c, k));
        };
        // like degrees side by side: a warp's threads then sum about as many records each
        std::sort(parts.begin() + b, parts.begin() + e, [&](uint32_t x, uint32_t y) {
            const uint32_t tx = inc[1]->ranges[x].y, ty = inc[1]->ranges[y].y;
            if (tx != ty) return tx > ty;
            const uint32_t ex = inc[0]->ranges[x].y, ey = inc[0]->ranges[y].y;
            return ex != ey ? ex > ey : x < y;
        });
        for (uint32_t i = 0; i < p; ++i) {
            stamp[parts[b + i]] = mark;
            localOf[parts[b + i]] = i;
        }
        // record slots in slices of 32 particles (the last one narrower): record q of a slice's
        // particle j at base + q * width + j, so a warp's q-th records are adjacent
        uint32_t slots[2] = {0u, 0u};
        std::vector<uint32_t> rec[2];
        for (int f = 0; f < 2; ++f) {
            rec[f].resize(p);
            for (uint32_t s0 = 0; s0 < p; s0 += 32u) {
                const uint32_t width = std::min(32u, p - s0);
                uint32_t most = 0;
                for (uint32_t i = s0; i < s0 + width; ++i) {
                    const uint32_t cnt = inc[f]->ranges[parts[b + i]].y;
                    if (cnt > kTileMaxRecords || slots[f] + width > 0xfffeu) return false;
                    most = std::max(most, cnt);
                    rec[f][i] = tileRecord(slots[f] + (i - s0), width, cnt);
                }
                slots[f] += most * width;
                if (slots[f] > 0xfffeu) return false;
            }
        }
        halo.clear();
        for (int f = 0; f < 2; ++f) {
            ids[f].clear();
            for (uint32_t i = b; i < e; ++i) {
                const uint2 r = inc[f]->ranges[parts[i]];
                for (uint32_t q = r.x; q < r.x + r.y; ++q) {
                    const uint32_t c = inc[f]->inc[q].x;
                    if (entryStamp[f][c] == mark) continue;
                    entryStamp[f][c] = mark;
                    ids[f].push_back(c);
                    for (uint32_t k = 0; k < per[f]; ++k) {
                        const uint32_t x = elem(f, c, k);
                        if (x >= n || stamp[x] == mark) continue;
                        stamp[x] = mark;
                        halo.push_back(x);
                    }
                }
            }
        }
        const size_t pos = size_t(p) + halo.size();
        if (pos > 0xffffu) return false;
        size_t need[2];
        for (int f = 0; f < 2; ++f) {
            need[f] = pos * 16 + size_t(slots[f]) * 12;
            if (need[f] > cap) return false;
        }
        std::sort(halo.begin(), halo.end());
        for (uint32_t k = 0; k < halo.size(); ++k) localOf[halo[k]] = p + k;
        // Entries of like shape (the same steps between their particles' local indices) side by side,
        // ascending in the first particle: on a lattice a warp's threads then read neighbouring positions
        // and write neighbouring record slots, free of bank conflicts.
        for (int f = 0; f < 2; ++f) {
            order.clear();
            for (uint32_t c : ids[f]) {
                uint32_t l[4] = {0u, 0u, 0u, 0u};
                for (uint32_t k = 0; k < per[f]; ++k) {
                    const uint32_t x = elem(f, c, k);
                    l[k] = x < n ? localOf[x] : 0u;
                }
                const uint64_t shape = uint64_t((l[1] - l[0]) & 0xffffu) << 32 | uint64_t((l[2] - l[0]) & 0xffffu) << 16 |
                                       uint64_t((l[3] - l[0]) & 0xffffu);
                order.push_back({shape, l[0], c});
            }
            std::sort(order.begin(), order.end());
            for (uint32_t k = 0; k < order.size(); ++k) {
                ids[f][k] = std::get<2>(order[k]);
                entryOf[f][ids[f][k]] = k;
            }
        }

        TileHead h{};
        h.own = uint32_t(out.own.size());
        h.ownCount = p;
        h.halo = uint32_t(out.halo.size());
        h.haloCount = uint32_t(halo.size());
        h.bends = bends ? 1u : 0u;
        for (int f = 0; f < 2; ++f) {
            h.entry[f] = uint32_t(out.id[f].size());
            h.entryCount[f] = uint32_t(ids[f].size());
            h.slots[f] = slots[f];
            out.smem[f] = std::max(out.smem[f], uint32_t(need[f]));
            out.id[f].insert(out.id[f].end(), ids[f].begin(), ids[f].end());
            out.rec[f].insert(out.rec[f].end(), rec[f].begin(), rec[f].end());
        }
        out.own.insert(out.own.end(), parts.begin() + b, parts.begin() + e);
        out.halo.insert(out.halo.end(), halo.begin(), halo.end());
        for (uint32_t c : ids[0]) {
            const uint32_t a = localOf[elem(0, c, 0)], z = localOf[elem(0, c, 1)];
            out.edges.push_back(make_uint2(a | (z << 16), 0xffffffffu));
        }
        for (uint32_t c : ids[1]) {
            uint32_t l[4];
            for (uint32_t k = 0; k < 4; ++k) {
                const uint32_t x = elem(1, c, k);
                l[k] = x < n ? localOf[x] : 0u;
            }
            out.elems.push_back(make_uint4(l[0] | (l[1] << 16), l[2] | (l[3] << 16), 0xffffffffu, 0xffffffffu));
        }
        for (int f = 0; f < 2; ++f)
            for (uint32_t i = 0; i < p; ++i) {
                const uint2 r = inc[f]->ranges[parts[b + i]];
                const uint32_t base = tileRecordBase(rec[f][i]), width = tileRecordWidth(rec[f][i]);
                for (uint32_t q = 0; q < r.y; ++q) {
                    const uint2 ck = inc[f]->inc[r.x + q];
                    const uint32_t at = h.entry[f] + entryOf[f][ck.x], slot = base + q * width;
                    uint32_t &word = f == 0 ? out.edges[at].y : (ck.y < 2u ? out.elems[at].z : out.elems[at].w);
                    const uint32_t shift = 16u * (ck.y & 1u);
                    word = (word & ~(0xffffu << shift)) | (slot << shift);
                }
            }
        out.heads.push_back(h);
        return true;
    }

    const In &in;
    std::vector<uint32_t> &parts;
    const size_t cap;
    std::vector<uint32_t> localOf, stamp;
    std::vector<uint32_t> entryOf[2], entryStamp[2];
    std::vector<uint32_t> ids[2], halo;
    std::vector<std::tuple<uint64_t, uint32_t, uint32_t>> order;
    uint32_t attempt = 0;
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
    // the lists take ~1.5 us a particle on one thread: one for every 2,048 particles, up to 16
    const uint32_t workers = std::min({std::max(in.n / 2048u, 1u), std::max(std::thread::hardware_concurrency(), 1u), 16u});
    for (uint8_t c = 1; c <= 2; ++c) {
        std::vector<uint32_t> parts;
        for (uint32_t i = 0; i < in.n; ++i)
            if (in.cls[i] == c) parts.push_back(i);
        if (parts.empty()) continue;
        // recursive bisection into leaves of equal size, in depth-first order
        const uint32_t count = uint32_t(parts.size()), tiles = (count + target - 1u) / target;
        auto split = [&](auto &&self, uint32_t b, uint32_t e, uint32_t t, uint32_t threads) -> std::vector<Leaf> {
            if (t <= 1u || e - b <= 1u) return {Leaf{b, e}};
            const uint32_t left = t / 2u, mid = Builder::bisect(in, parts, b, e, left, t);
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
            Builder b(in, parts, smemCap);
            for (size_t l = leaves.size() * k / shares; l < leaves.size() * (k + 1u) / shares; ++l)
                b.leaf(leaves[l].begin, leaves[l].end, c == 2);
            built[k] = std::move(b.out);
        });
        for (TileBuild &t : built) {
            if (!t.ok) return TileBuild{};
            for (TileHead &h : t.heads) {
                h.own += uint32_t(out.own.size());
                h.halo += uint32_t(out.halo.size());
                for (int f = 0; f < 2; ++f) h.entry[f] += uint32_t(out.id[f].size());
            }
            auto append = [](auto &to, const auto &from) { to.insert(to.end(), from.begin(), from.end()); };
            append(out.heads, t.heads);
            append(out.own, t.own);
            append(out.halo, t.halo);
            append(out.edges, t.edges);
            append(out.elems, t.elems);
            for (int f = 0; f < 2; ++f) {
                append(out.rec[f], t.rec[f]);
                append(out.id[f], t.id[f]);
                out.smem[f] = std::max(out.smem[f], t.smem[f]);
            }
        }
    }
    out.ok = !out.heads.empty();
    return out;
}

} // namespace cn
