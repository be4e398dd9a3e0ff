// Rules of the host side that depend on sizes alone: how work is divided.  No CUDA in here, so that a test can compile
// and check them without a GPU.
#pragma once

namespace dmm {

// How many CTAs share the tiles of the wide kernel that are left over from the whole ones (`rest` of them, of `units` units and
// `nb` columns each), and whether the contributors of a split tile add its parts up together (dmm_wide.cuh, share_fixup).
struct WideSplit {
    long long parts;  // rest: one whole tile per CTA
    bool share;
};
// Shared where the parts of a tile are this many KiB or more; below the last CTA is done sooner by itself, the sharing costs
// it some 1.5 us of atomics.  us at the same split, alone / shared, means of all measured splits by KiB: 75 to 100 + 0.4 us, 125 to
// 150 - 0.2, 175 to 200 - 0.7, 300 - 2.1, 600 - 4.  64 x 4096 x 11008 (576 KiB) 26.4 / 22.4, 64 x 4096 x 4096 16.9 / 14.1, 33 x 8192 x 8192 (222 KiB)
// 22.6 / 22.0, 33 x 14336 x 2048 with 148 CTAs (127 KiB) 21.4 / 23.5.  Only in the 64-column build: up to 32 columns there is less to
// read (8 x 4096 x 4096 9.6 / 10.9), and at 128 the second form of the fix-up cost the kernel registers (500 x 4096 x 4096 37.6 / 41.3).
constexpr long long kWShareKiB = 150;

inline WideSplit wide_split(int nb, int units, long long rest, int num_sms, bool can_split, bool atomic) {
    // Estimated cycles of the longest CTA.  A unit costs about 640 + 10 nb, and a split tile a fix-up: its last CTA reads nb KiB
    // per contributor at 64 bytes a cycle.  (An estimate that ranks the splits well, not the rate: in the steady state a unit takes
    // 1080 cycles up to 32 columns and 1480 at 128.)  A shared fix-up is estimated like one that is not: it is faster at any
    // number of contributors, but with every one of them it gets slower all the same (each piece is summed over all parts by
    // one warp).  Taken for a flat cost it led small matrices to more CTAs than pay: us with the flat cost / now, 33 rows 16 x 32768
    // (148 / 20 CTAs) 43.4 / 20.0, 1024 x 4096 (128 / 32) 19.6 / 12.5, 4096 x 1024 (128 / 16, whole tiles) 11.8 / 8.2, 64 rows 512 x 8192 33.4 / 15.0.
    WideSplit s = {rest, false};
    long long best = 0;
    for (long long c = rest; can_split && c <= num_sms; c = c < num_sms && c + rest > num_sms ? num_sms : c + rest) {
        if (c > rest && c > rest * units) break;
        const long long n = (rest * units + c - 1) / c, contributors = c == rest ? 0 : (c + rest - 1) / rest + 1;
        const long long fix = contributors == 0 ? 0 : 3000 + 16ll * nb * (atomic ? 1 : contributors + 1);
        const long long cost = n * (640 + 10 * nb) + fix;
        if (best == 0 || cost < best) {
            best = cost;
            s.parts = c;
        }
    }
    s.share = s.parts > rest && !atomic && nb > 32 && nb <= 64 && nb * s.parts >= kWShareKiB * rest;
    return s;
}

// Batch 1 and 2: four k-tiles per hand-over instead of two (PolF8Long) from 28 tiles per segment on.  The longer hand-over
// gains with every tile and loses some 0.2 us at the end of each segment, where nothing is left to decode beside the MMAs
// of the last one.  A CTA has about 1 + super-tiles / SMs segments.  PolF8 / PolF8Long in us, batch 1, added into a stack, and
// tiles per segment: 57344 x 512 6.81 / 7.32 (10), 4096 x 4096 5.17 / 5.45 (13), 40960 x 1024 7.58 / 7.88 (17), 57344 x 1024 8.64 / 8.88
// (19), 16384 x 2048 6.57 / 6.75 (19), 6144 x 6144 6.70 / 6.82 (27), 11008 x 4096 7.58 / 7.56 (29; a result of its own 10.93 / 10.82),
// 57344 x 2048 13.14 / 13.13 (39), 8192 x 8192 9.11 / 9.00 (45), 28672 x 8192 20.6 / 20.1 (110).
struct HandoverSize {
    long long tiles = 0, segments = 0, sms = 0;  // of all CTAs; SMs of all products
    long long silu_tiles = 0;                    // those of the products behind silu(gate) * up
    void add(long long N, long long K, int num_sms, bool silu) {
        const long long sst = (N + 255) / 256;
        tiles += sst * (K / 32);
        if (silu) silu_tiles += sst * (K / 32);
        segments += sst + num_sms;
        sms += num_sms;
    }
    int k_tiles() const { return tiles >= 28 * segments ? 4 : 2; }
    long long tiles_per_sm() const { return tiles / sms; }
};

// Whether the activations of a chunk of M <= 32 rows are split into planes once, by a kernel in front of the product, or by
// the product's own loaders in every CTA.  The kernel in front is one more dependent launch, 2 to 3 us; the loaders' split
// costs nothing up to 3 rows and then more with every row and tile, hence a number of tiles per SM for each row count.  us per
// block of a stack, planes / loaders, and its products' mean tiles per SM: 4 rows 41.2 / 34.7 (42), 49.0 / 42.5 (65), 86.8 / 83.1 (176);
// 5 rows 41.7 / 35.2, 49.3 / 44.0, 87.5 / 86.9; 6 rows 41.9 / 36.2, 49.5 / 47.7, 86.2 / 94.5; 7 rows 42.3 / 37.4, 50.0 / 49.0,
// 88.3 / 101.5; 8 rows 42.6 / 39.2, 50.4 / 51.0, 88.9 / 107.9.  The lines lie where straight lines through these met before the loaders'
// first epoch grew.  One plain product by itself still gains at its line, us, fp32 activations: 4 rows 43008 x 8192 (290) 31.2 / 30.5, 5 rows 20480 x
// 8192 (138) 18.1 / 17.1, 6 rows 11264 x 8192 (76) 13.0 / 12.1, 8 rows 8448 x 8192 (57) 11.7 / 11.1; launched one after the other, where
// the kernel in front waits for nothing, it is level there: 32.4 / 32.7, 19.4 / 19.0, 14.2 / 14.3, 12.8 / 13.2.
// Behind silu(gate) * up the loaders of every super-tile repeat the exponential, and what is one product of four in a block decides
// by itself: us per product, planes / loaders, launched programmatically 4 rows t = 41 10.3 / 9.6, 110 15.7 / 15.6, 290 32.2 / 34.8, 5 rows t = 138 18.2 / 20.3,
// 8 rows t = 37 10.3 / 10.4, 57 11.7 / 13.1; one after the other 4 rows t = 27 10.1 / 9.7, 55 12.5 / 12.7, 110 16.9 / 17.6, 6 rows t = 13 9.1 / 7.9, 20 9.9 / 10.2, 8 rows
// t = 20 10.1 / 10.5.  The lines are those at which neither way loses.
constexpr long long kPlanesMinBatch = 4;
constexpr int kPlanesMost[9] = {0, 0, 0, 0, 290, 144, 77, 63, 58}, kPlanesMostSilu[9] = {0, 0, 0, 0, 40, 16, 16, 16, 16};
inline bool planes_in_front(long long M, const HandoverSize &size) {
    if (M < kPlanesMinBatch || M > 8) return M > 8;
    return size.tiles_per_sm() > (2 * size.silu_tiles > size.tiles ? kPlanesMostSilu : kPlanesMost)[M];
}

// The same for the tensor-parallel products; mode as in UmmaParams.  A consumer of the slots form (3) splits what it sums up
// itself, and the kernel of its build with planes in turn with the one without costs more than planes gain: its producer (2) keeps
// to the plain lines whatever its input.  us per block in a group of one, planes from 4 rows on / so: 2048 wide 4 rows 43.6 / 36.5, 5 rows
// 48.0 / 39.3, 8 rows 50.2 / 41.8, 4096 wide 8 rows 75.1 / 69.7, 8192 wide 4 rows 127.6 / 124.5, 8 rows 172.1 / 172.2 (before there were
// two builds: 42.6, 46.1, 50.0, 76.8, 133.0, 177.7).  Products that add into every rank's buffer (0): planes from 4 rows on.
inline bool planes_in_front_tp(long long M, int mode, const HandoverSize &alone) {
    if (mode == 0) return M >= kPlanesMinBatch;
    return mode == 2 && M >= kPlanesMinBatch && (M > 8 || alone.tiles_per_sm() > kPlanesMost[M]);
}

}  // namespace dmm
