#pragma once
// Launch geometry shared by the collide kernels and the host code that
// sizes their grids.
#include <algorithm>

// Resident CTAs per SM the collide kernels are compiled for (sets the
// register cap: 65536 / (256 * this)).
#ifndef PFLBM_COLLIDE_MIN_BLOCKS
#define PFLBM_COLLIDE_MIN_BLOCKS 2
#endif

// Column tile of the collide kernels (x fastest; TX a multiple of 32).
#ifndef PFLBM_TILE_X
#define PFLBM_TILE_X 32
#endif
#ifndef PFLBM_TILE_Y
#define PFLBM_TILE_Y 8
#endif

namespace pflbm {
constexpr int kTileX = PFLBM_TILE_X, kTileY = PFLBM_TILE_Y;
static_assert(kTileX % 32 == 0 && kTileX * kTileY <= 1024, "collide tile");

// Interior planes per CTA of a z-marching collide launch over `tiles` column
// tiles and `nzi` interior planes, on `sms` SMs that hold `per_sm` of its CTAs
// each. Short chunks pay the warm-up of a CTA (four phi planes, two normal
// planes, an empty pipeline) over and over; the wrong number of chunks leaves
// most of the chip idle behind a few last CTAs. The time is modelled in planes
// of a full SM: a wave of full SMs takes the chunk and one and a half planes
// of warm-up that the neighbours on the SM do not hide; the last, partial wave
// takes as long on an SM with all its CTAs, half as long with a single one
// (which has the SM for itself), and hides less (two planes more). Of the
// chunks within 6% of the least, the one nearest to 8 planes is taken: what
// the model calls equal is faster with shorter chunks, whose CTAs read the
// planes more nearly in order. (Not always: the D3Q27 FP32 128x128x512 jet gets
// 20 planes instead of 27, 364 instead of 358 us.) Against the fastest of a
// sweep of chunks the choice is 1% slower on average over the 22 grids it was
// fitted on, 32x32x64 to 256x256x1024 (every storage type, plain and closure
// kernels; 4% at most), and over 36 random ones that it was not fitted on, up
// to 16 M nodes, 1.6% in FP32 (10% at most) and 4.8% in 16 bits (23% at most:
// D3Q19 BF16 97x165x33, 33 instead of 27 us). Eight CTAs per SM at least four
// planes long, the rule before: FP16 256x256x1024 1859 -> 1494 us, FP32
// 64x64x128 30.6 -> 22.6, 96^3 46.5 -> 33.1, 128^3 87.1 -> 71.0, of which a
// fifth to a third is the shorter warm-up.
inline int pick_zchunk(int tiles, int nzi, int sms, int per_sm) {
    auto planes = [&](int chunks) { return (nzi + chunks - 1) / chunks; };
    auto time = [&](int zc) {
        const long long n = 1ll * tiles * ((nzi + zc - 1) / zc), slots = 1ll * sms * per_sm;
        double t = double(n / slots) * (zc + 1.5);
        const long long rem = n % slots;
        if (rem > 0) {
            const int on = int((rem + sms - 1) / sms);  // CTAs on the fullest SM
            t += (per_sm > 1 ? 0.5 + 0.5 * (on - 1) / (per_sm - 1) : 1.0) * (zc + 1.5) + (on < per_sm ? 2 : 0);
        }
        return t;
    };
    double least = 1e300;
    for (int chunks = 1; chunks <= nzi && (planes(chunks) >= 2 || chunks == 1); ++chunks)
        least = std::min(least, time(planes(chunks)));
    int best = nzi;
    double off = 1e300;
    for (int chunks = 1; chunks <= nzi && (planes(chunks) >= 2 || chunks == 1); ++chunks) {
        const int zc = planes(chunks);
        const double d = zc > 8 ? zc / 8.0 : 8.0 / zc;
        if (time(zc) <= 1.06 * least && d <= off) off = d, best = zc;
    }
    return std::max(best, 1);
}
}  // namespace pflbm
