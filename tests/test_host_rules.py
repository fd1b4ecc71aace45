"""Rules that size and route launches, as host arithmetic: compiled from the library's own headers and checked over their
whole range without a GPU."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "rknpu2_matmul_open_b200" / "csrc"


def _run(tmp_path, body):
    (tmp_path / "rule.cpp").write_text(body)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", f"-I{CSRC}", "-o", str(tmp_path / "rule"), str(tmp_path / "rule.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "rule")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_expert_rows_are_read_inside_the_piece_that_holds_them(tmp_path):
    # the intake kernel requests an fp32 row for every block of its grid, whether the run has that row or not
    _run(tmp_path, r"""
#include "moe_rows.h"
#include <initializer_list>
#include <stdio.h>
using namespace rkb200;
#define CHECK(x) do { if (!(x)) { printf("%s: H %d max_rows %d rows %d f32 %d\n", #x, H, most, rows, f32); return 1; } } while (0)
int main()
{
    for (int H : {64, 96, 512, 544, 1024, 1536, 1984, 2048, 2400, 4064, 4096, 7168, 8128, 8192})
        for (int most = 1; most <= 256; ++most)
            for (int f32 = 0; f32 < 2; ++f32) {
                int grid[2][9] = {};
                for (int rows = 1; rows <= most; ++rows) {
                    const MoeRowPlan p = moe_row_plan(rows, most, H, f32);
                    const size_t bytes = size_t(f32 ? 4 : 1) * H, piece = moe_piece_row_bytes(most, H);
                    CHECK(p.grid_rows >= rows && p.grid_rows <= most && p.level >= 0 && p.level <= 8);
                    CHECK(!p.pull || rows * bytes <= piece);                       // what the host stages
                    CHECK(!p.pull || !f32 || p.grid_rows * bytes <= piece);       // what the kernel may request
                    int& kept = grid[p.pull][p.level];                            // the launches of a kind are kept
                    CHECK(kept == 0 || kept == p.grid_rows);
                    kept = p.grid_rows;
                }
            }
    return 0;
}
""")


def test_results_that_the_kernel_stores_over_the_bus(tmp_path):
    # sizes at which copying and storing were both measured; the faster one is the rule's
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int family, M, cols, elem; bool store; };
int main()
{
    const Case cases[] = {
        {5, 4, 4911, 4, true}, {5, 3, 7001, 2, true}, {5, 4, 14330, 4, true}, {5, 8, 4911, 4, true}, {5, 8, 14331, 4, true}, {5, 1, 4911, 2, true},
        {3, 8, 2900, 2, true}, {3, 8, 2900, 4, true}, {3, 8, 28672, 4, true}, {3, 8, 9984, 4, true},
        {3, 8, 4911, 2, false}, {3, 8, 9998, 4, false}, {3, 5, 14330, 2, false}, {3, 8, 40000, 4, false},
        {1, 13, 4912, 2, true}, {1, 13, 4910, 2, false}, {2, 64, 1024, 2, true}, {2, 64, 2048, 2, false},
    };
    for (const Case& c : cases)
        if (result_over_bus(c.family, c.M, size_t(c.cols), size_t(c.elem)) != c.store) { printf("family %d %d x %d x %d\n", c.family, c.M, c.cols, c.elem); return 1; }
    return 0;
}
""")


def test_rows_that_leave_the_single_launch_at_mid_batches(tmp_path):
    # the faster of the two forms where both were measured and differ by more than 3 %
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int M, K; bool half, ring; };
int main()
{
    const Case cases[] = {
        {9, 4096, true, false}, {16, 4096, true, false}, {16, 1024, true, false}, {9, 1500, true, false}, {12, 2044, true, true}, {16, 3070, true, true},
        {16, 1025, true, true}, {9, 4096, false, false}, {9, 1024, false, false}, {13, 4096, false, true}, {16, 2048, false, true}, {16, 8192, false, true},
        {9, 2044, false, true}, {9, 3070, false, true}, {12, 1500, false, true}, {9, 1025, false, true},
    };
    for (const Case& c : cases)
        if (mid_batch_takes_ring(c.M, c.K, c.half) != c.ring) { printf("%d x %d half %d\n", c.M, c.K, c.half); return 1; }
    return 0;
}
""")


def test_tiles_in_parts_are_launched_whatever_can_be_resident(tmp_path):
    # a plan is made for half of the SMs in pairs; where fewer pairs can be resident its parts still all run
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
int main()
{
    for (int resident = 1; resident <= 76; ++resident)
        for (int tiles = 1; tiles <= 200; ++tiles)
            for (int split = 1; split <= 8; ++split) {
                const int clusters = persist_clusters(tiles, split, resident);
                if (split > 1 ? clusters != tiles * split : clusters < 1 || clusters > resident || clusters > tiles || (clusters < resident && clusters != tiles)) {
                    printf("%d tiles in %d parts, %d resident: %d\n", tiles, split, resident, clusters);
                    return 1;
                }
            }
    return 0;
}
""")


def test_runs_of_items_cover_every_token_of_every_channel_tile_once(tmp_path):
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
#include <vector>
using namespace rkb200;
int main()
{
    for (int tiles : {1, 2, 5, 16, 43, 56, 112, 300})
        for (int per_tile : {1, 2, 3, 4, 5, 7, 24, 25, 64, 94, 128})
            for (int most = 1; most <= 8; ++most)
                for (int snap : {0, 2, 3})
                    for (int pairs : {1, 2, 37, 73, 74}) {
                        const int units = tiles * per_tile;
                        const int n = persist_clusters(units, 1, pairs);
                        std::vector<char> seen(units, 0);
                        bool ok = true;
                        for (int i = 0; i < n; ++i) {
                            const unsigned from = persist_bound(units, per_tile, snap, i, n), to = persist_bound(units, per_tile, snap, i + 1, n);
                            ok = ok && from <= to && (i || from == 0) && (i + 1 < n || to == (unsigned)units);
                            PersistItems items(from, to, per_tile, most);
                            int tile, first, len;
                            while (items.next(tile, first, len)) {
                                ok = ok && tile >= 0 && tile < tiles && first >= 0 && len >= 1 && len <= most && first + len <= per_tile;
                                for (int k = 0; ok && k < len; ++k) ok = !seen[tile * per_tile + first + k]++;
                            }
                        }
                        for (char c : seen) ok = ok && c == 1;
                        if (!ok) { printf("%d tiles of %d, most %d, snap %d, %d pairs\n", tiles, per_tile, most, snap, pairs); return 1; }
                    }
    return 0;
}
""")


def test_runs_of_very_many_units(tmp_path):
    # one channel tile of 2^31 tokens is 2^26 units: runs begin in order and cover all of them, and the plan, made for every
    # memory query, does not take longer for it; its stretches of equal items are the items that the kernel walks
    _run(tmp_path, r"""
#include "persist_plan.h"
#include <initializer_list>
#include <stdio.h>
#include <time.h>
#include <vector>
using namespace rkb200;
int main()
{
    for (unsigned units : {57456230u, 58000000u, 67108864u, 2147483647u, 4294967295u})
        for (unsigned per_tile : {1u, 7u, 57456230u, 67108864u, 4294967295u})
            for (unsigned snap : {0u, 3u})
                for (unsigned pairs : {1u, 2u, 66u, 74u, 75u, 1600u}) {
                    unsigned from = 0;
                    for (unsigned i = 0; i < pairs; ++i) {
                        const unsigned exact = (unsigned)((unsigned long long)units * i / pairs), at = persist_bound(units, per_tile, snap, i, pairs);
                        if (at < from || (snap == 0 && at != exact)) { printf("run %u of %u over %u: %u\n", i, pairs, units, at); return 1; }
                        from = at;
                    }
                    if (persist_bound(units, 1, snap, pairs, pairs) != units) return 2;
                }
    for (int M : {4096, 100000000, 2000000000, 2147483647})
        for (int columns : {1, 300, 2147483647}) {
            const clock_t before = clock();
            for (int kind = 0; kind < 3; ++kind) persist_plan(columns, M, 1, kind == 1, kind == 2, 148);
            if (clock() - before > CLOCKS_PER_SEC / 20) { printf("a plan for %d tokens, %d columns took %g s\n", M, columns, double(clock() - before) / CLOCKS_PER_SEC); return 3; }
        }
    struct Walked { int first, units; };
    for (unsigned per_tile : {1u, 2u, 5u, 13u, 24u})
        for (unsigned most = 1; most <= 8; ++most)
            for (unsigned begin = 0; begin <= 2 * per_tile; ++begin)
                for (unsigned end = begin; end <= 4 * per_tile; ++end) {
                    std::vector<Walked> walked, told;
                    PersistItems items(begin, end, per_tile, most);
                    for (int tile, first, n; items.next(tile, first, n);) walked.push_back({first, n});
                    persist_stretches(begin, end, per_tile, [&](unsigned first, unsigned len, unsigned tiles) {
                        while (tiles--) {
                            unsigned at = first;
                            persist_widths(len, most, [&](unsigned units, unsigned n) { for (; n--; at += units) told.push_back({(int)at, (int)units}); });
                            if (at != first + len) told.clear();
                        }
                    });
                    bool same = walked.size() == told.size();
                    for (size_t i = 0; same && i < walked.size(); ++i) same = walked[i].first == told[i].first && walked[i].units == told[i].units;
                    if (!same) { printf("units %u to %u, %u a tile, most %u\n", begin, end, per_tile, most); return 4; }
                }
    return 0;
}
""")


def test_cuts_that_the_gpu_tests_force(tmp_path):
    # accepted as they are; every width of an item is among them, some runs begin or end inside a channel tile, and some pair takes
    # more items than there are accumulators
    from persist_cuts import GRIDS, LONG, LONG_FFN, PARTS, RUNS, WHOLE, WHOLE_FFN
    cuts = [f"{{{M}, {K}, {N}, {{{cut}}}}}" for shapes, names in (((WHOLE, WHOLE_FFN), GRIDS + RUNS), ((LONG, LONG_FFN), PARTS))
            for M, K, N in shapes for cut in names]
    _run(tmp_path, r"""
#include "persist_plan.h"
#include <stdio.h>
#include <set>
using namespace rkb200;
struct Cut { int M, K, N; PersistPlan plan; };
int main()
{
    const Cut cuts[] = {CUTS};
    const PersistPlan refused[] = {{0, 1, 0, 1}, {48, 1, 0, 1}, {288, 1, 0, 1}, {64, 2, 0, 1}, {32, 9, 0, 1}, {32, 2, 4, 1}, {32, 1, 0, 0}, {32, 1, 0, 9},
                                   {192, 1, 0, 2}, {32, 2, 0, 2}, {32, 1, 0, 8}, {-32, 1, 0, 1}, {32, -1, 0, 1}, {32, 0, 0, 1}};
    for (const PersistPlan& p : refused)
        if (persist_cut_ok(p, 31)) { printf("%d,%d,%d,%d accepted\n", p.unit, p.most, p.snap, p.split); return 1; }
    std::set<int> of_one_width, of_runs;
    int inside = 0;
    for (const Cut& c : cuts) {
        const PersistPlan& p = c.plan;
        if (!persist_cut_ok(p, (c.K + 127) / 128)) { printf("%d,%d,%d,%d refused\n", p.unit, p.most, p.snap, p.split); return 2; }
        if (p.split > 1) continue;
        const unsigned per_tile = (c.M + p.unit - 1) / p.unit, units = (c.N + 255) / 256 * per_tile, pairs = persist_clusters(units, 1, 74);
        const int accumulators = p.unit * p.most > PS_WIDE ? 1 : 2;
        int longest = 0;
        for (unsigned i = 0; i < pairs; ++i) {
            const unsigned from = persist_bound(units, per_tile, p.snap, i, pairs);
            PersistItems items(from, persist_bound(units, per_tile, p.snap, i + 1, pairs), per_tile, p.most);
            inside += from % per_tile != 0;
            int n_items = 0;
            for (int tile, first, n; items.next(tile, first, n); ++n_items) (p.most > 1 ? of_runs : of_one_width).insert(n * p.unit);
            if (n_items > longest) longest = n_items;
        }
        if (longest <= accumulators) { printf("%d,%d,%d,%d: %d items a pair\n", p.unit, p.most, p.snap, p.split, longest); return 3; }
    }
    return of_one_width.size() == 8 && of_runs.size() == 8 && inside ? 0 : 4;
}
""".replace("CUTS", ", ".join(cuts)))


def test_families_for_few_tokens(tmp_path):
    # sizes at which the three families were measured, within 7 % of the fastest; every answer is a family that shares the layout
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int M, K, cols; bool half; int family; };
int main()
{
    const Case cases[] = {
        {1, 4096, 4096, true, 5}, {1, 1024, 14336, true, 3}, {1, 11008, 2048, true, 3}, {2, 4096, 6144, true, 5}, {2, 5120, 5120, false, 3},
        {2, 8192, 8192, false, 1}, {3, 11008, 8192, true, 5}, {4, 8192, 2048, false, 3}, {4, 4096, 6144, true, 3}, {4, 8192, 8192, true, 1},
        {4, 3070, 4911, true, 1}, {4, 4096, 4096, false, 5}, {4, 5120, 13824, false, 1}, {5, 2048, 4096, true, 5}, {5, 5120, 5120, false, 3},
        {8, 2048, 2048, false, 5}, {8, 4096, 4096, true, 3}, {8, 4096, 4096, false, 1}, {8, 2048, 14336, true, 1}, {8, 4096, 11008, true, 3}, {4, 4096, 11008, true, 5}, {4, 2048, 5632, true, 5}, {3, 3584, 7680, true, 5}, {3, 5120, 5632, true, 3}, {8, 3070, 4911, false, 1},
        {8, 8192, 1024, false, 3}, {8, 8192, 2048, false, 1}, {6, 8192, 2048, false, 3}, {5, 1500, 2048, true, 5}, {8, 1500, 2048, true, 5}, {3, 3072, 8192, false, 3}, {4, 11008, 8192, false, 5},
    };
    for (const Case& c : cases) {
        const int from = c.M <= 4 || (long long)c.K * c.cols / 2 > (24 << 20) ? 5 : 3;
        if (few_tokens_linear(from, c.M, c.K, c.cols, c.half) != c.family) { printf("%d x %d -> %d half %d\n", c.M, c.K, c.cols, c.half); return 1; }
    }
    for (int M = 1; M <= 8; ++M)
        for (int K = 1; K < 20000; K += 37)
            for (int cols = 1; cols < 40000; cols += 401)
                for (int bit = 0; bit < 2; ++bit)
                    for (int from = 3; from <= 5; from += 2) {
                        const int f[2] = {few_tokens_linear(from, M, K, cols, bit), few_tokens_ffn(from, M, K, cols, bit)};
                        for (int x : f) if (x != 1 && x != 3 && x != 5) { printf("%d x %d -> %d: %d\n", M, K, cols, x); return 1; }
                    }
    for (int M = 9; M <= 16; ++M)
        if (!mid_batch_call_takes_ring(M, 4096, 4096, true, false) || mid_batch_call_takes_ring(M, 4096, 4096, true, true) || !mid_batch_call_takes_ring(M, 4096, 2048, false, true) ||
            mid_batch_call_takes_ring(9, 1024, 300, true, false)) { printf("%d\n", M); return 1; }
    return 0;
}
""")


def test_ctas_of_a_cluster_that_share_the_quantisation(tmp_path):
    # units of 16 elements a token; fp32 rows of one token were measured up to 12288 elements, with and without a partner
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int M, units; bool half; int ctas; };
int main()
{
    const Case cases[] = {{1, 576, false, 1}, {1, 688, false, 1}, {1, 768, false, 1}, {1, 776, false, 4}, {1, 768, true, 1}, {1, 896, true, 4}, {2, 512, false, 1}, {2, 768, false, 4},
                          {2, 768, true, 1}, {4, 768, true, 1}, {4, 768, false, 4}, {8, 512, true, 1}, {8, 768, true, 4}, {8, 576, false, 4}};
    for (const Case& c : cases)
        if (decode_cluster(c.M, c.units, c.half) != c.ctas) { printf("%d tokens, %d units, half %d\n", c.M, c.units, c.half); return 1; }
    return 0;
}
""")


def test_families_for_few_tokens_where_the_ring_is_thin(tmp_path):
    # sizes on both sides of the rounds of the ring, the clusters and the decode kernel: no slower than the workspace's own family and
    # within 10 % of the fastest of the three
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int M, K, cols; bool half; int family; };
int main()
{
    const Case cases[] = {
        {1, 8192, 11008, true, 5}, {1, 8192, 12416, true, 5}, {1, 8192, 14336, true, 1}, {1, 11008, 8192, false, 1}, {1, 6144, 22016, true, 5},
        {2, 4096, 11008, false, 5}, {2, 4096, 12544, false, 5}, {2, 4096, 14336, false, 1}, {2, 4096, 18944, false, 5}, {2, 5120, 6912, false, 1}, {2, 5120, 9984, false, 1},
        {2, 6144, 9216, false, 5}, {2, 5888, 11664, false, 1}, {2, 4825, 8385, false, 1}, {2, 5120, 6144, true, 1}, {2, 5120, 5120, true, 3}, {2, 10752, 4608, true, 5}, {2, 8192, 9216, true, 5},
        {3, 4096, 7168, false, 1}, {3, 11008, 6144, true, 5}, {3, 10112, 5693, true, 3}, {3, 5120, 9984, false, 1}, {4, 4096, 12544, false, 1}, {4, 4096, 18944, false, 5}, {4, 4096, 18944, true, 5},
        {4, 2048, 40960, false, 5}, {4, 6144, 11008, true, 1}, {4, 6144, 18944, true, 5}, {5, 4405, 1792, true, 3}, {6, 4702, 1024, true, 3}, {5, 4405, 6000, true, 1}, {6, 11008, 6144, false, 1},
        {8, 4096, 8320, true, 1}, {8, 4096, 11776, true, 3}, {8, 4096, 12288, true, 1}, {8, 4096, 12544, true, 1}, {8, 4096, 14336, true, 1}, {8, 4096, 28672, true, 1},
        {5, 4608, 11008, true, 1}, {5, 5120, 9984, true, 5}, {8, 6144, 9216, true, 5}, {8, 8192, 11008, true, 5}, {8, 8192, 14336, true, 1}, {5, 1664, 7168, true, 1}, {8, 1664, 4736, true, 5}, {8, 3072, 4736, true, 3}, {8, 3072, 4864, true, 1}, {6, 4224, 6272, true, 1}, {8, 2048, 22528, true, 1}, {8, 1024, 28672, true, 1}, {8, 1024, 49152, true, 3},
    };
    for (const Case& c : cases) {
        const int from = c.M <= 4 || (long long)c.K * c.cols / 2 > (24 << 20) ? 5 : 3;        // the workspace's
        const int family = few_tokens_linear(from, c.M, c.K, c.cols, c.half);
        if (family != c.family) { printf("%d x %d -> %d half %d: %d\n", c.M, c.K, c.cols, c.half, family); return 1; }
    }
    return 0;
}
""")


def test_first_projections_where_the_ring_is_thin(tmp_path):
    # columns: two a feature; no slower than the decode kernel, which is the workspace's own, and no slower than the ring by more than 5 %
    # where K is at least 5120 or up to 3328
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int M, K, cols, family; };
int main()
{
    const Case cases[] = {
        {1, 8192, 14336, 1}, {1, 8192, 18944, 5}, {2, 5120, 22016, 1}, {2, 6144, 18944, 5}, {4, 4096, 22016, 5}, {5, 3072, 22016, 1}, {5, 3584, 18944, 5}, {8, 4096, 22016, 5}, {5, 5120, 18944, 5},
        {5, 6144, 9216, 1}, {8, 6144, 22016, 5}, {8, 8192, 11008, 1}, {5, 8192, 18944, 5}, {8, 8192, 22016, 5}, {8, 5120, 27648, 1}, {8, 3840, 4992, 1},
    };
    for (const Case& c : cases)
        if (few_tokens_ffn(5, c.M, c.K, c.cols, false) != c.family) { printf("%d x %d -> %d\n", c.M, c.K, c.cols); return 1; }
    return 0;
}
""")


def test_calls_of_nine_to_sixteen_tokens(tmp_path):
    # both sides of the lines between one launch and two: 256 KB of weights, few channels of long rows, collected maxima with up to 2112 channels
    _run(tmp_path, r"""
#include "w4a8_rules.h"
#include <stdio.h>
using namespace rkb200;
struct Case { int M, K, cols; bool half, collected, ring; };
int main()
{
    const Case cases[] = {
        {9, 1024, 512, true, false, false}, {9, 1024, 520, true, false, true}, {16, 1024, 512, true, false, false}, {13, 1024, 512, false, false, true}, {12, 1024, 512, false, false, false},
        {12, 1500, 300, true, false, true}, {10, 1500, 300, true, false, false}, {9, 4096, 4096, true, false, true}, {16, 2048, 8192, false, false, true},
        {12, 11008, 1024, true, false, false}, {12, 11008, 1024, false, false, false}, {13, 11008, 1024, true, false, true}, {12, 8192, 1024, true, false, true}, {12, 11008, 1056, true, false, true},
        {9, 4096, 2112, false, true, true}, {16, 4096, 2113, false, true, false}, {12, 11008, 1024, false, true, false}, {16, 11008, 1024, false, true, true}, {9, 512, 64, false, true, true},
    };
    for (const Case& c : cases)
        if (mid_batch_call_takes_ring(c.M, c.K, c.cols, c.half, c.collected) != c.ring) { printf("%d x %d -> %d half %d collected %d\n", c.M, c.K, c.cols, c.half, c.collected); return 1; }
    return 0;
}
""")
