// w4a8_rules.h -- rules of the W4A8 dispatch that are plain arithmetic on sizes.  Host only, no CUDA.
#pragma once
#include <stddef.h>

#include "persist_plan.h"

namespace rkb200 {

// Whether a blocking call's kernel stores its [M][cols] result of `elem` bytes each straight into page-locked host memory
// instead of leaving it to the copy engine.  `family`: the kernel family that runs the call (5 decode, 3 split-K, others in
// two launches).
//   * The decode kernel writes every element once, 32 neighbouring ones per warp: rows that do not start on a sector cost it
//     nothing visible (4 x 4911 fp32 26 us against 33 copied, 4 x 14330 32 against 38, 8 x 4911 at K = 11008 47 against 55).
//   * The split-K kernel stores four neighbours at once where the row length allows it (8 x 2900 binary16 26 us against 32
//     copied); element by element the bus takes them slowly (8 x 4911 58 us against 33), so then small results only.
//   * The single-kernel families up to 1 MB (8 x 28672 fp32 44 us against 49, into an ordinary array 84 against 100).  The
//     others write pieces of 64 bytes, which the bus takes more slowly: from 128 KB on the copy engine is as fast, and rows
//     that do not start on a sector leave it in pieces of sectors (13 x 4910 binary16 64 us against 38, 13 x 4912 34).
constexpr size_t RESULT_OVER_BUS_MOST = size_t(1) << 20;
inline bool result_over_bus(int family, int M, size_t cols, size_t elem)
{
    const size_t bytes = size_t(M) * cols * elem;
    const bool single = family == 5 || family == 3;
    if (bytes > (single ? RESULT_OVER_BUS_MOST : size_t(128) << 10)) return false;
    if (M == 1 || family == 5 || cols * elem % 32 == 0 || (family == 3 && cols % 4 == 0)) return true;
    return bytes <= (elem == 2 ? size_t(40) << 10 : size_t(64) << 10);
}

// Cluster size of the decode kernel (= how many CTAs share the quantisation) for `units` of 16 elements, token slots included.
// Quantising a unit costs a thread about 500 cycles of issue slots and the exchange about as much as one and a half units, so up to
// three units per thread stay local; beyond that four CTAs share (clusters of eight leave half of this GPU's SMs without a CTA).  fp32
// rows are twice the loads and the higher token slots more work per unit: two units (8 x 1536 -> 4096 fp32 6.4 us with 768, 5.3; binary16
// 5.5 and 5.3; at 3072 -> 8192 with 4 tokens of binary16 the exchange costs more, 6.5 with 768 and 7.7).  A single row is little either
// way, and CTAs with several groups of channels wait for each other: fp32 11008 -> 6144 14.4 with 768, 16.1 with 512, -> 11008 19.2 and 21.1.
inline int decode_cluster(int M, long long units, bool half) { return units <= (M == 1 || (half && M <= 4) ? 768 : 512) ? 1 : 4; }

// CTAs (of a cluster) that share a column tile of the ring: the smallest number that gives nearly every SM a CTA.  More only adds
// reduction traffic and shortens each CTA's stream, and more than 33 clusters of eight or 66 of four need not be resident at once (two
// CTAs an SM, whole clusters in a GPC), which costs a second round.  (Until every SM had one: 34 tiles in eight parts, 12 x 4096 ->
// 4352 10.5 us, in four 7.4; 72 tiles in four parts, 8 x 4096 -> 9152 11.2, in two 8.5; 65 tiles, 8 x 4096 -> 8320, in four 7.0, in
// two 8.7.)
inline int ring_parts(long long tiles, int KB, int sms)
{
    int parts = 1;
    while (parts < 8 && tiles * parts * 10 < sms * 9ll && KB / (parts * 2) >= 2) parts *= 2;
    return parts;
}

constexpr int RULE_SMS = 148;

// How much of its rounds a launch fills: `ctas` of equal work, `places` at once.
inline double filled(long long ctas, long long places) { return double(ctas) / double((ctas + places - 1) / places * places); }

// The ring's CTAs, `parts` of K for each column tile, two an SM.  Where the last round leaves more than three eighths of the places
// empty, SMs with one CTA stream with half of their bandwidth: 4096 -> 14336, 224 CTAs, 9.5 us, -> 18944, 148 CTAs, 14.9.  In four
// parts and more a CTA's stream is short and that costs little.
struct RingFill {
    int parts;
    double used;
    bool fills, thin;
    RingFill(int K, int columns, int sms)
    {
        const long long tiles = (columns + 127ll) / 128;
        parts = ring_parts(tiles, (K + 127) / 128, sms);
        used = filled(tiles * parts, 2 * sms);
        fills = used >= 0.625;
        thin = !fills && parts <= 2;
    }
};

// Up to eight tokens: the family that runs a call of a workspace of family 3 (split-K clusters) or 5 (decode); the code layout is the
// ring's (1) too.  Measured on 33 shapes of both types and again on 146, the times are of one call of a back-to-back series in us, decode / clusters /
// ring.  The two single launches scan and quantise the rows in every cluster, the ring has a launch of its own for that and costs 6.3
// at least: long rows, large weights and rows without 16-byte loads are the ring's (8 x 4096 -> 4096 fp32 7.8 / 7.9 / 6.5,
// 4 x 8192 -> 8192 13 / 12.6 / 10.6, 8 x 3070 -> 4911 10.3 / 13.2 / 7.6).  The decode kernel's CTAs take 32 channels over all of K:
// best on short rows (8 x 2048 -> 2048 5.2 / 5.7 / 6.2), poor on few channels of long rows (4 x 8192 -> 2048 8.5 / 6.4 / 7.2) and
// where some CTAs have two groups of channels (4 x 5120 -> 5120 9.0 / 7.0 / 7.9).
inline int few_tokens_linear(int family, int M, int K, int columns, bool half, int sms = RULE_SMS)
{
    const double mb = double(K) * columns / 2 / (1 << 20);          // of weights
    const bool ragged = K % (half ? 8 : 4) != 0;
    const int groups = int((columns + 31ll) / 32);
    const RingFill ring(K, columns, sms);
    // The clusters hold their weights in shared memory: on 148 SMs a CTA has one column tile up to 12.5 MB (fused_tiles_per_cta) and
    // two beyond, and from about 28 MB on they are not resident at once (3 x 11008 -> 6144 11.5 / 22.4 / -, 6 fp32 17.2 / 25.0 / -).
    const bool one_tile = mb * RULE_SMS <= 12.5 * sms, one_round = mb * RULE_SMS <= 28. * sms;
    if (M > 4) {
        if (K <= 3072 && mb <= 4.5) return 5;
        if (ragged) return half && M <= 6 && K >= 4096 && mb <= 11.2 ? 3 : 1;       // 5 x 4405 -> 1792 8.4 / 7.4 / 8.3, -> 6000 12.7 / 10.6 / 9.7
        if (half) {
            // 8 x 3072 -> 8192 9.0 / 7.1 / 7.0, 2048 -> 14336 8.9 / 9.7 / 6.9, 4096 -> 8320 9.5 / 9.7 / 7.6.  Where the ring is thin:
            //   * 5 x 6144 -> 9216 11.1 / 13.1 / 12.8, 8 x 8192 -> 11008 15.0 / 26.7 / 15.8, 4608 -> 11008 13.8 / 12.4 / 10.3;
            //   * the clusters are near alone and in front in a chain (4096 -> 11008 11.7 / 10.1 / 9.3, layers of 4096 / 11008 with 8 tokens
            //     65.9 / 61.3 / 62.7, of 4096 / 11776 65.5 / 61.4 / 63.3); beyond they are not (4096 -> 12288 11.8 / 12.6 / 9.4, -> 14336
            //     13.8 / 13.8 / 9.7, layers of 4096 / 14336 70.7 / 73.4 / 65.2); short rows are quantised sooner (2048 -> 22528 11.8 / 10.2 / 9.0).
            // With a second round of channel groups the ring is in front alone and in a chain (5 x 1664 -> 7168 6.7 / 6.5 / 5.6, 8 x 3072 -> 8192
            // 8.7 / 7.4 / 6.7, -> 4096 6.8 / 6.7 / 6.0; layers of 1664 / 7168 with 5 tokens 39.1 / 41.7 / 37.0, of 3072 / 8192 48.4 / 47.3 / 46.4).
            if (mb <= 13.25) return groups > sms ? 1 : family;
            if (ring.thin && K >= 5120) return 5;
            return mb > 20 && family == 3 && (K <= 1280 || (K > 3072 && K <= 4096 && ring.thin)) ? 3 : 1;    // 8 x 1024 -> 49152 15.8 / 9.5 / 11.2
        }
        if (columns <= 1024 || (K >= 8192 && columns <= 2112 && M <= 6)) return 3;
        return M <= 6 && one_tile && groups > 144 && groups <= 192 ? 3 : 1;
    }
    if (columns <= 2112 && (K >= 8192 || (K >= 6144 && (M > 1 || !half)))) return 3;
    // (In a chain of binary16 calls 3 x 3584 -> 7680, 240 groups, takes the decode kernel 1 less; 4 x 4096 -> 6144, 192 groups, the clusters
    // 1.4.)  fp32: 3 x 4096 -> 7168 8.3 / 9.4 / 6.9
    if ((half && M > 2 ? one_round && K < 10240 : one_tile) && groups > 144 && groups <= (half ? 192 : 240) && !ragged && M > 1 && K > (M == 2 ? 4096 : 3072)) return 3;
    if (!half && (one_tile || (ragged && M == 3 && mb < 14)) && groups > 144 && groups <= 296 && M > 2 && K >= 3072) return 3;      // 4 x 3072 -> 8192 7.7 / 6.7 / 6.5
    if (K <= 1024 && groups > 296) return 3;                         // 4 x 1024 -> 14336 6.1 / 5.6 / 6.3
    if (ragged && M == 4 && mb > 4) return 1;
    if (M > 2) {
        // 4 x 6144 -> 11008 14.0 / 13.6 / 12.5, 4 x 8192 -> 9216 15.8 / 22.9 / 14.4; in one part 4 x 6144 -> 18944 17.9 / 24.8 / 21.1
        const bool pays = ring.fills || (K >= 4608 && ring.parts > 1);
        // (in a chain 4 x 4096 -> 11008 of binary16 takes the decode kernel 0.9 less than the ring)
        if (half) return mb >= 14 && K <= 8192 && (mb >= 26 || K >= 6144) && pays ? 1 : family;
        // long rows of 112 to 148 groups stay: 3 x 11008 -> 4096 9.1 / 10.9 / 9.1 alone, in a layer the ring is 4 behind
        return !ragged && !one_tile && K < 10240 && pays ? 1 : family;
    }
    // Two tokens cost the decode kernel less: fp32 4096 -> 11008 8.6 / 9.5 / 9.2, -> 12544 8.8 / 10.8 / 9.3, -> 14336 10.5 / 11.2 / 9.4,
    // 5120 -> 6912 9.8 / 9.4 / 7.6, binary16 5120 -> 6144 8.6 / 9.6 / 7.5; where the ring is thin it is behind unless the decode kernel's
    // last round is as empty (fp32 5120 -> 9216, 288 groups, 10.5 / 9.8 / 10.9, -> 11008, 344 groups, 12.9 / 11.8 / 11.0).
    const double decode_used = filled(groups, sms);
    const bool better = ring.fills || decode_used < 0.85;
    if (M == 2) {
        if (half && mb >= 14 && K >= 8192 && !ring.thin && better) return 1;
        if (half && !one_tile && groups > sms && groups <= 192 && !ragged && K > 4096) return 1;
        if (!half && mb >= 14 && (K >= 5120 || (ragged && K >= 4096)) && better) return 1;
        if (!half && mb >= 28 && K >= 4096 && ring.fills) return 1;
        return mb >= 40 && !ring.thin ? 1 : family;
    }
    // One token: 8192 -> 11008 14.0 / 22.4 / 15.6, -> 12416 14.2 / - / 15.6, -> 14336 17.0 / - / 15.7, 11008 -> 8192 13.6 / - / 12.5
    return mb >= 40 && ring.used > 0.9 * decode_used ? 1 : family;
}

// The same for the two projections of an FFN (times of the whole FFN).  The first's columns come in pairs and its quantising is fp32
// (2048 -> 2 x 14336, 4 tokens: 22.9 / - / 17.9); the second finds its rows' maxima collected, so no kernel scans (14336 -> 1024
// behind it 19.9 / 17.9 / 19.6, 5632 -> 2048 at 4 tokens 16.1 / 14.9 / 15.0).
inline int few_tokens_ffn(int family, int M, int K, int columns, bool second, int sms = RULE_SMS)
{
    const double mb = double(K) * columns / 2 / (1 << 20);
    if (second) {
        if (M <= 4) return columns <= 2112 && K >= 5120 ? 3 : family;
        if (mb <= 2) return 5;
        return columns <= 2112 && K <= 6144 ? 1 : family;
    }
    if (K <= 2048 && columns > 2 * 32 * sms) return columns < 16384 && M <= 4 ? 3 : 1;
    if (K % 4 && M >= 4) return 1;
    // The ring's one part is slow where it is thin, on longer rows above all: 5 x 3072 -> 2 x 11008 23.0 and 20.6, but 5120 -> 2 x 9472 23.7 and
    // 26.9, 8192 -> 2 x 9472 29.5 and 36.3, 1 x 8192 -> 2 x 9472 27.1 and 35.1; in two parts 5 x 6144 -> 2 x 4608 19.6 and 19.5.
    const RingFill ring(K, columns, sms);
    const bool pays = ring.fills || ring.parts > 1;
    if (M <= 2 && mb >= 50 && (M == 2 || K >= 8192) && (pays || K <= 5120)) return 1;       // 1 x 8192 -> 2 x 7168 27.6 / - / 25.1
    if (M <= 4) return family;
    // 8 x 3840 -> 2 x 2496 -> 3840 with the decode kernel in front 18.0, with the ring 15.5 (clusters 16.6); 2560 -> 2 x 6912 18.7 and
    // 15.9, 5120 -> 2 x 3456 17.7 and 16.3; but 2048 -> 2 x 5632 14.3 and 14.4, 4096 -> 2 x 5504 17.7 and 18.1, 4096 -> 2 x 11008 25.3 and 27.7
    return K > 2048 && (K < 4096 || K >= 5120) && (pays || K < 3328) ? 1 : 5;
}

// 9..16 tokens of very small weights: whether one launch (the split-K kernel, whose every cluster scans all of the rows) is left for
// two (quantise, ring): fp32 rows are twice the scan, rows that are loaded element by element sooner still.
inline bool mid_batch_takes_ring(int M, int K, bool half)
{
    const bool wide = K % 8 == 0;
    return half ? !wide && M > 10 : M > (wide ? 12 : 8);
}

// 9..16 tokens of a workspace of family 3: whether a call takes two launches (quantise, ring) instead of the split-K kernel, whose
// every cluster scans all of the rows.  Always but for weights of 256 KB, where a launch is most of the work, and unless the rows'
// maxima are there already and the channels many (4096 -> 4096 behind a first projection: the FFN 19.4 us with one launch, 20.3 with
// two; 4096 -> 2048 16.9 and 14.6).  16 tokens binary16, 1024 -> 1024 7.6 us with one and 6.5 with two, 4096 -> 4096 9.8 and 7.5;
// fp32 2048 -> 8192 12.2 and 6.6.
inline bool mid_batch_call_takes_ring(int M, int K, int columns, bool half, bool maxima_collected)
{
    const bool long_rows = columns <= 1024 && K > 8192 && M <= 12;   // 10 x 11008 -> 1024 fp32 9.3 us with one, 9.8 with two
    if (maxima_collected) return columns <= 2112 && !long_rows;
    return (!long_rows && (long long)K * columns / 2 > (256ll << 10)) || mid_batch_takes_ring(M, K, half);
}

} // namespace rkb200
