// persist_plan.h -- how a launch of the persistent GEMM (w4a8_gemm_tc_persist.cu) is cut into items: the dealing, which every role
// of the kernel walks on the GPU, and the plan, made on the host once for a workspace.  Arithmetic on sizes; needs no CUDA.
#pragma once
#include <algorithm>
#include <math.h>
#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define RKB200_HD __host__ __device__ __forceinline__
#else
#define RKB200_HD inline
#endif

namespace rkb200 {

constexpr int PERSIST_T = 1;            // tokens of a group of activation codes (GemmParams::T): every token's codes lie in one piece
constexpr int PERSIST_TOKENS = 32;      // the code buffer holds a whole multiple of these, items are multiples of them

// The widest item of a kernel that takes the plan's.  (int8 weights: the first and the last.)
constexpr int PS_NARROW = 64, PS_WIDE = 160, PS_WIDEST = 256;

// How a problem is cut (columns: all accumulator rows, i.e. gate and up together for SwiGLU): pairs of channel tiles x units of
// tokens, dealt to the CTA pairs in runs.
struct PersistPlan {
    int unit;     // tokens, a multiple of 32
    int most;     // units of an item
    int snap;     // see persist_bound
    int split;    // parts K is cut into; one item per launch unit then, and most is 1
};

// Whether the kernel runs a cut: one of those that persist_plan chooses from, whatever it would choose.
inline bool persist_cut_ok(const PersistPlan& cut, int KB)
{
    const bool grid = cut.most == 1 && cut.snap == 0 && cut.unit % PERSIST_TOKENS == 0, runs = cut.unit == PERSIST_TOKENS && cut.most > 1 && cut.snap >= 0 && cut.snap <= 3;
    if (!(grid || runs) || cut.unit < PERSIST_TOKENS || cut.most > PS_WIDEST / PERSIST_TOKENS || cut.unit > PS_WIDEST || cut.split < 1 || cut.split > 8) return false;
    return cut.split == 1 || (grid && cut.unit <= PS_WIDE && KB >= 4 * cut.split);
}

// CTA pairs of a launch: one per part where tiles are cut along K (no part waits for another, the last to arrive finishes the
// tile, so more pairs than are resident at once run in turn), else at most as many as can be resident, each with a run of items.
inline int persist_clusters(int tiles, int split, int resident)
{
    if (split > 1) return tiles * split;
    return tiles < resident ? tiles : resident;
}

// A channel tile's tokens are counted in units; all units of all channel tiles, one tile's behind the other's, are dealt to
// the CTA pairs in equal runs: run i begins at units * i / pairs.  Where a run would begin or end less than `snap` units from the
// edge of a channel tile, the edge is taken: a narrow item costs nearly as much as a wide one.  The host divides by the pairs,
// before anything is multiplied: nothing here is larger than `units`, and the rounded-up inverse is exact for rest * i * pairs
// below 2^32, i.e. up to 1600 pairs.  (64-bit divisions on the GPU cost a launch of K = 1024 a microsecond.)
struct PersistShare {
    unsigned whole, rest;       // units / pairs and what is left
    unsigned inverse;           // 2^32 / pairs, rounded up (0 for one pair, which has no rest)
};
inline PersistShare persist_share(unsigned units, unsigned pairs)
{
    return {units / pairs, units % pairs, unsigned(((uint64_t(1) << 32) + pairs - 1) / pairs)};
}
RKB200_HD unsigned persist_bound(PersistShare share, unsigned per_tile, unsigned snap, unsigned i)
{
    const unsigned x = share.whole * i + (unsigned)(((uint64_t)(share.rest * i) * share.inverse) >> 32), in = x % per_tile;
    if (in && in < snap) return x - in;
    if (in && per_tile - in < snap) return x + per_tile - in;
    return x;
}
inline unsigned persist_bound(unsigned units, unsigned per_tile, unsigned snap, unsigned i, unsigned pairs)
{
    return persist_bound(persist_share(units, pairs), per_tile, snap, i);
}

// The items of one run, in order: what lies in one channel tile is cut into as few items of at most `most` units as
// possible, of nearly equal width.
struct PersistItems {
    unsigned tile, first;       // where the next item begins: channel tile, unit inside it
    unsigned left_units;        // of the run
    unsigned per_tile, most;
    unsigned pieces, seg_end;   // items left in this channel tile, and their end inside it
    RKB200_HD PersistItems(unsigned begin, unsigned end, unsigned units_per_tile, unsigned most_units)
        : tile(begin / units_per_tile), first(begin - begin / units_per_tile * units_per_tile), left_units(end - begin), per_tile(units_per_tile), most(most_units), pieces(0), seg_end(0) {}
    // channel tile, first unit inside it and units of the next item; false: there is none
    RKB200_HD bool next(int& in_tile, int& at, int& units)
    {
        if (!left_units) return false;
        if (!pieces) {
            seg_end = first + left_units < per_tile ? first + left_units : per_tile;
            pieces = most == 1 ? seg_end - first : (seg_end - first + most - 1) / most;
        }
        const unsigned n = most == 1 ? 1 : (seg_end - first + pieces - 1) / pieces;
        in_tile = (int)tile;
        at = (int)first;
        units = (int)n;
        first += n;
        left_units -= n;
        if (--pieces == 0 && first == per_tile) { first = 0; ++tile; }
        return true;
    }
};

// The same items without walking them: visit(units of an item, how many of them follow each other, whether the tile ends with
// them) for `len` units of one channel tile, and for a run visit(first unit inside the tile, units, how many tiles alike).
template <class Visit>
inline void persist_widths(unsigned len, unsigned most, Visit visit)
{
    const unsigned pieces = (len + most - 1) / most, wider = pieces ? len % pieces : 0;
    if (wider) visit(len / pieces + 1, wider);
    if (pieces) visit(len / pieces, pieces - wider);
}
template <class Visit>
inline void persist_stretches(unsigned begin, unsigned end, unsigned per_tile, Visit visit)
{
    if (const unsigned in = begin % per_tile; in && begin < end) {
        const unsigned head = std::min(end - begin, per_tile - in);
        visit(in, head, 1u);
        begin += head;
    }
    if (const unsigned tiles = (end - begin) / per_tile) visit(0u, per_tile, tiles);
    if (const unsigned tail = (end - begin) % per_tile) visit(0u, tail, 1u);
}

// The cheapest cut by a model of a call's time, fitted to every cut of 709 linears and 244 int8-weight calls (1 to 3000 tokens,
// K 1024 .. 11008, 1024 .. 14336 channels; SwiGLU launches: an earlier fit, which 319 shapes bear out).  Only what cuts of one
// shape differ by was fitted, so the constants are the fit's cycles, not the kernel's.  What it takes costs 0.5 to 0.9 % against
// the best cut in the mean:
//   * a k-block of an item costs a constant (the issuer's and the unpack warps' chains) and something per token, so wide items
//     pay; less where SMs are idle, a little more in runs, whose pairs do not share weights;
//   * finishing an item is hidden behind the next one's MMAs (two accumulators) unless it takes longer.  Rows whose length does
//     not allow four channels in one store cost 9 % more of it per token (2 to 3 % of a call at a fixed cut; when they were priced
//     at two and a half times, 512 x 4096 -> 4911 took 22.4 us for 20.0 and 2266 x 4032 -> 1285 26.9 for 24.5);
//   * K in parts costs an exchange through L2: so much per part and pair, more for wide items;
//   * a launch that leaves too few SMs free has the next call's quantise kernel wait for it, and its own set-up for that kernel: no
//     cost up to `knee` of the pairs, counting `rows` of them per thousand tokens to quantise, all of it `ramp` further
//     (109 x 4352 -> 4547 14.7 us on 72 pairs, 13.4 on 36).
// A run is priced by its stretches of equal items, so that a plan takes the same few microseconds whatever the token count.
struct PersistCosts {
    double narrow, narrow_token, wide, wide_token, widest, widest_token;   // a k-block in each kernel
    double finish, finish_token, ragged, item;       // finishing an item (per token so many times as much for ragged rows), and between two
    double part0, part, pair, part_wide;             // the exchange of parts
    double crowded, knee, ramp, rows;                // see above
    double idle, runs;                               // of a k-block: less with idle pairs, so many times as much in runs
};
// Cycles a cut takes; `enough`: more than that need not be told exactly.  (columns and tokens whose units fit 31 bits)
inline double persist_cut_cycles(const PersistCosts& cost, const PersistPlan& cut, int columns, int M, int KB, bool w8, int pairs, double enough)
{
    const int unit = cut.unit, most = cut.most, split = cut.split;
    const int64_t tokens = (int64_t(M) + PERSIST_TOKENS - 1) / PERSIST_TOKENS * PERSIST_TOKENS;
    const unsigned per_tile = unsigned((tokens + unit - 1) / unit), units = unsigned((int64_t(columns) + 255) / 256) * per_tile;
    const int clusters = persist_clusters(int(units), split, pairs);
    const double busy = std::min(1.0, double(clusters) / pairs), load = (1 - cost.idle * (1 - busy)) * (most > 1 ? cost.runs : 1);
    const bool narrow = unit * most <= PS_NARROW, wide = unit * most <= PS_WIDE, hidden = w8 || wide;
    auto block = [&](double width) {
        return load * (narrow ? cost.narrow + cost.narrow_token * width : wide ? cost.wide + cost.wide_token * width : cost.widest + cost.widest_token * width);
    };
    auto finish = [&](double width) { return cost.finish + cost.finish_token * (columns % 4 ? cost.ragged : 1) * width; };
    auto run = [&](unsigned begin, unsigned end) {
        double time = 0, last = 0;                       // `last`: finishing the item in front, not paid for yet
        auto alike = [&](double width, unsigned n) {
            const double mmas = KB * block(width) + cost.item, then = finish(width);
            time += hidden ? std::max(mmas, last) : mmas + last;
            time += (n - 1) * (hidden ? std::max(mmas, then) : mmas + then);
            last = then;
        };
        persist_stretches(begin, end, per_tile, [&](unsigned first, unsigned len, unsigned tiles) {
            const bool short_end = first + len == per_tile && int64_t(per_tile) * unit > tokens;    // (items of one unit then)
            auto tile = [&] {
                persist_widths(len, most, [&](unsigned n_units, unsigned n) {
                    if (n > short_end) alike(double(n_units) * unit, n - short_end);
                    if (short_end) alike(double(tokens - int64_t(per_tile - 1) * unit), 1);
                });
            };
            tile();
            if (tiles == 1) return;
            const double so_far = time;
            tile();
            time += (tiles - 2) * (time - so_far);
        });
        return time + last;
    };
    double longest = 0;
    if (split > 1) {
        const double width = double(std::min<int64_t>(unit, tokens));
        longest = KB * block(width) / split + finish(width) +
                  (cost.part0 + cost.part * (split - 1) + cost.pair * clusters) * (1 + cost.part_wide * std::max(0.0, width - 64) / 64.0);
    } else {
        const PersistShare dealt = persist_share(units, unsigned(clusters));
        for (int i = 0; i < clusters && longest < enough; ++i)
            longest = std::max(longest, run(persist_bound(dealt, per_tile, cut.snap, i), persist_bound(dealt, per_tile, cut.snap, i + 1)));
    }
    return longest + cost.crowded * std::min(1.0, std::max(0.0, (busy + cost.rows * M / 1000 - cost.knee) / cost.ramp));
}
inline const PersistCosts& persist_costs(bool w8, bool swiglu)
{
    static const PersistCosts linear{349, 2.48, 415, 1.53, 351, 2.15, 3000, 41.1, 1.09, 138, 1860, 1640, 8.33, 1.38, 2340, 0.569, 0.0642, 0.314, 0.316, 1.02};
    static const PersistCosts gated{366, 0.79, 420, 0.37, 326, 1.0, 5060, 60, 2.5, 670, 1500, 1380, 30, 0.7, 2030, 0.5, 0.01, 0, 0.15, 1};
    static const PersistCosts bytes{355, 2.58, 506, 1.75, 474, 2.08, 5070, 52, 1.75, 709, 4210, 1510, 16.3, 0.976, 989, 0.782, 0.121, 0.0751, 0.107, 1};
    return w8 ? bytes : swiglu ? gated : linear;
}
// Every cut that is considered: visit(cut).
template <class Visit>
inline void persist_cuts(int columns, int M, int KB, int pairs, Visit visit)
{
    const int64_t channel_tiles = (int64_t(columns) + 255) / 256, tokens = (int64_t(M) + PERSIST_TOKENS - 1) / PERSIST_TOKENS * PERSIST_TOKENS;
    const int widest = int(std::min<int64_t>(PS_WIDEST, tokens));
    for (int unit = PERSIST_TOKENS; unit <= widest; unit += PERSIST_TOKENS)       // items of one width, K in parts or not
        for (const int split : {1, 2, 3, 4, 6, 8}) {
            if (split > 1 && (unit > PS_WIDE || channel_tiles * ((tokens + unit - 1) / unit) * split > pairs || KB < 4 * split)) break;
            visit(PersistPlan{unit, 1, 0, split});
        }
    for (int most = 2; most <= widest / PERSIST_TOKENS; ++most)                  // equal runs
        for (const int snap : {0, 2, 3}) visit(PersistPlan{PERSIST_TOKENS, most, snap, 1});
}
inline PersistPlan persist_plan(int columns, int M, int KB, bool w8, bool swiglu, int sm_count)
{
    PersistPlan best{PERSIST_TOKENS, 1, 0, 1};
    if ((int64_t(columns) + 255) / 256 * ((int64_t(M) + PERSIST_TOKENS - 1) / PERSIST_TOKENS) > INT32_MAX) return best;   // (its activations or results fit no GPU)
    const PersistCosts& cost = persist_costs(w8, swiglu);
    const int pairs = std::max(1, sm_count / 2);
    double best_cycles = HUGE_VAL;
    persist_cuts(columns, M, KB, pairs, [&](const PersistPlan& cut) {
        const double cycles = persist_cut_cycles(cost, cut, columns, M, KB, w8, pairs, best_cycles);
        if (cycles < best_cycles) { best_cycles = cycles; best = cut; }
    });
    return best;
}

} // namespace rkb200
