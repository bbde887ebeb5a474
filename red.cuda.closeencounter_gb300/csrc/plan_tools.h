// plan_tools.h -- host-side launch-plan helpers shared by the single-disk and the ensemble
// plans (header-only, no CUDA types: the CPU tests compile it alone).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <utility>
#include <vector>

namespace redgb {

// The FP64 kernel of a block with more sources than the row-serial kernel takes (64): `rows` sinks and
// `pairs` (sink, source) pairs, over all systems of an ensemble.
//   rows (grav_fp64_rows): a CTA per row, 304 resident, 4.4 us a wave up to some 200 sources
//   pair-parallel (grav_fp64_pairpar): S sinks a CTA; 30 to 45 ps a pair
//   certified (grav_fp64_cert): 25 us more, then 2.7 ns a row of up to a few hundred sources
// Square blocks go by their pairs: self-interacting blocks of 400 / 1000 / 1300 / 1480 bodies on
// GB300: rows 18 / 55 / 85 / 101 us, certified 48 / 88 / 99 / 109 us; of 1700 and 2000, before the
// rows' last gain of a tenth, rows 146 / 195 us, certified 124 / 149 us.  Wide, shallow ones by their
// rows: those of 65 / 103 / 203 / 403 sources go pair by pair from 510 / 650 / 1070 / 2160 sinks (an
// evaluation of 65 massive bodies and 5000 test particles: 85 us in rows, 23 pair by pair, 68
// certified; an RKF7(8) attempt of 5 disks of 403 bodies 974 us in rows, 1088 pair by pair, of 12 1971
// and 1736), certified from some 240 000 / 28 000 / 8400 / 3500 (203 and 20 000: 189 us pair by pair, 117
// certified; 12 disks of 303 bodies 868 us pair by pair, 1219 certified, of 30 2071 and 1330).
enum Fp64Form { FP64_FORM_ROWS, FP64_FORM_PAIRPAR, FP64_FORM_CERT };
constexpr int64_t FP64_ROW_PAIRS = 2250000;
inline bool fp64_wide(int64_t rows, int64_t pairs)
{
    const int64_t src = rows > 0 ? pairs / rows : 0;
    return 1000 * rows > 300000 + 3000 * src + 4 * src * src;
}
inline Fp64Form fp64_block_form(int64_t rows, int64_t pairs)
{
    if (!fp64_wide(rows, pairs)) return pairs <= FP64_ROW_PAIRS ? FP64_FORM_ROWS : FP64_FORM_CERT;
    return pairs - 60 * rows <= 1200000 ? FP64_FORM_PAIRPAR : FP64_FORM_CERT;  // rows (sources - 60)
}

// The sinks S of a pair-parallel CTA for the blocks added: 256 threads take four terms each of S x
// 1024 / S pairs at a time, `resident` CTAs on each of n_sm SMs.  The S of the least waves x steps (a
// CTA starts and sums for as long as two steps of terms take; two thirds of a wave's rounding count: an
// evaluation of 203 massive bodies and 2000 test particles takes 39 us with 8 and 54 with 16, with
// 5000 82 and 73; 64 disks of 103 bodies 565 us an attempt with 8, 529 with 16, 661 with 32).
struct PairparSinks {
    static constexpr int S[4] = {4, 8, 16, 32};
    double ctas[4] = {}, steps[4] = {};
    void add(int sinks, int sources)
    {
        for (int k = 0; k < 4; k++) {
            const int stride = 256 / S[k], tile = 4 * stride, n = (sinks + S[k] - 1) / S[k];
            ctas[k] += n;
            steps[k] += (double)n * (sources / tile * 4 + (sources % tile + stride - 1) / stride + 2);
        }
    }
    int best(int resident, int n_sm) const
    {
        int s = 8;
        double least = -1.0;
        for (int k = 0; k < 4; k++) {
            if (ctas[k] <= 0.0) continue;
            const double waves = ctas[k] / ((double)resident * std::max(n_sm, 1));
            const double cost = (2.0 * std::ceil(waves) + std::max(1.0, waves)) * steps[k] / ctas[k];
            if (least < 0.0 || cost < least) {
                least = cost;
                s = S[k];
            }
        }
        return s;
    }
};

// How long `sink_tiles` tiles of sinks take in source chunks of `tiles` of `src_tiles` source tiles each,
// in source tiles: the CTAs, all whole chunks and then the last, shorter ones, go one after the
// other to the slot that is free first, and a CTA starts for as long as a third of a source tile takes.
constexpr double MIXED_START_COST = 0.3;
inline double mixed_chunk_time(int sink_tiles, int src_tiles, int tiles, int slots)
{
    const int chunks = (src_tiles + tiles - 1) / tiles;
    const int64_t whole = (int64_t)sink_tiles * (chunks - 1);
    const double d = tiles + MIXED_START_COST, last = src_tiles - (chunks - 1) * tiles + MIXED_START_COST;
    const int64_t waves = whole / slots, over = whole % slots;
    // [time, slots free from then on], earliest first
    std::vector<std::pair<double, int64_t>> free = {{waves * d, slots - over}};
    if (over) free.push_back({(waves + 1) * d, over});
    double end = (waves + (over ? 1 : 0)) * d;
    int64_t left = sink_tiles;
    for (size_t k = 0; left > 0; k++) {
        const std::pair<double, int64_t> f = free[k];
        const int64_t n = std::min(left, f.second);
        left -= n;
        end = std::max(end, f.first + last);
        const std::pair<double, int64_t> next{f.first + last, n};
        free.insert(std::upper_bound(free.begin() + (ptrdiff_t)k + 1, free.end(), next), next);
    }
    return end;
}

// Source chunks (grid.y) of the mixed tile kernel, two CTAs to an SM, for `sink_tiles` tiles of
// sinks and `src_tiles` tiles of sources: as many as fit in one wave of CTAs, or, where that
// leaves fewer, enough for 16 waves in chunks of at least six source tiles (a CTA starts with its
// sinks and the heavy sources, so shorter chunks repeat more of that; a grid of one to three
// waves leaves the chip to the last of them).  Evaluations on GB300, one chunk per about 4 CTAs
// an SM -> this rule: 1001 bodies 43.7 -> 28 us, 3001 60.5 -> 36 us, 16 385 358 -> 319 us,
// 131 074 16.56 -> 15.7 ms.
// Where the six tiles leave one to three waves, the count of the least mixed_chunk_time (the fewest on
// a tie) is taken if it is better by 15 %, which is about how far that time is to be trusted (no CTA
// runs alone on its SM in it, which is half as fast again): 6600 / 8500 / 9600 / 12 500 bodies
// 87 / 128 / 138 / 208 us with six tiles, 77 / 110 / 128 / 200 us so; 13 000 and 14 000 bodies would
// gain 14 and 5 % by it and lose 6.
inline int mixed_chunk_count(int sink_tiles, int src_tiles, int n_sm)
{
    const int64_t slots = 2 * (int64_t)std::max(n_sm, 1), tiles = std::max(sink_tiles, 1);
    const int64_t one_wave = slots / tiles;
    const int64_t many = std::min<int64_t>((16 * slots + tiles - 1) / tiles, src_tiles / 6);
    int best = (int)std::max<int64_t>(1, std::min<int64_t>(std::max(one_wave, many), src_tiles));
    if (src_tiles < 2) return best;
    const auto time_of = [&](int n) {
        return mixed_chunk_time((int)tiles, src_tiles, (src_tiles + n - 1) / n, (int)slots);
    };
    double least = time_of(best) / 1.15;
    for (int n = 1; n <= src_tiles; n++) {
        if (n > 1 && (src_tiles + n - 1) / n == (src_tiles + n - 2) / (n - 1)) continue;  // as with one chunk fewer
        const double t = time_of(n);
        if (t < least - 1e-9) {
            least = t;
            best = n;
        }
    }
    return best;
}

// Segments of the symmetric heavy-light kernel (grav_df_sym).  `systems` holds one tile per
// system: its light bodies [sink_begin, sink_end) (and whatever else the kernel reads, copied
// into every segment).  The kernel's CTA takes a segment in passes of `unit` bodies (one per
// thread), then reduces the segment's heavy-row sums, so a segment costs its passes plus a
// fixed `seg_cost` (in passes).  The light bodies of all systems, end to end, are cut into
// passes (a system's last one partial), and the passes into n_cta contiguous ranges of equal
// cost, a system's first pass carrying the segment cost; a range's pieces in different
// systems are its segments.  Appends the segments, each with its part of its system's heavy
// rows (from 1, in the order of its light bodies), to `tiles`; CTA c takes the segments
// [cta_seg[c], cta_seg[c + 1]) of those appended (n_cta + 1 entries); parts[k] = 1 + the
// segments of system k (the heavy-heavy part is part 0).
template <class TileT>
void build_sym_segments(const std::vector<TileT>& systems, int n_cta, int unit, double seg_cost,
                        std::vector<TileT>& tiles, std::vector<int>& cta_seg, std::vector<int>& parts)
{
    const size_t t0 = tiles.size();
    struct Pass {
        int sys, b0, b1;
        double cost;
    };
    std::vector<Pass> pass;
    double total = 0.0;
    for (size_t k = 0; k < systems.size(); k++)
        for (int b = systems[k].sink_begin; b < systems[k].sink_end; b += unit) {
            const double c = 1.0 + (b == systems[k].sink_begin ? seg_cost : 0.0);
            pass.push_back(Pass{(int)k, b, std::min(b + unit, systems[k].sink_end), c});
            total += c;
        }
    parts.assign(systems.size(), 1);
    cta_seg.clear();
    size_t q = 0;
    double done = 0.0;
    for (int c = 0; c < n_cta; c++) {
        cta_seg.push_back((int)(tiles.size() - t0));
        // this CTA's passes: up to the cost boundary (c + 1) total / n_cta, the pass that
        // crosses it going to the side nearer to it; the last CTA takes the rest
        const double goal = total * (c + 1) / n_cta;
        int prev_sys = -1;
        while (q < pass.size()) {
            const bool last = c == n_cta - 1;
            if (!last && done + pass[q].cost * 0.5 > goal) break;
            const Pass& p = pass[q];
            if (p.sys == prev_sys) {
                tiles.back().sink_end = p.b1;  // the same segment goes on
            } else {
                TileT t = systems[p.sys];
                t.sink_begin = p.b0;
                t.sink_end = p.b1;
                t.part = parts[p.sys]++;
                tiles.push_back(t);
                prev_sys = p.sys;
            }
            done += p.cost;
            q++;
        }
    }
    cta_seg.push_back((int)(tiles.size() - t0));
}

}  // namespace redgb
