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

}  // namespace dmm
