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
// of a full SM: a wave of full SMs takes the chunk and one plane of warm-up
// that the neighbours on the SM do not hide; the last, partial wave takes as
// long on an SM with all its CTAs, three quarters as long with a single one
// (which has the SM for itself), and hides less (four planes more). The chunk
// with the least is taken. Against the fastest of a sweep of chunks the choice
// is 1% slower on average over 22 grids from 32x32x64 to 256x256x1024 (every
// storage type, plain, averaging and closure kernels; 3% at most) and 2% over
// 36 random ones (17% at most). Eight CTAs per SM at least four planes long,
// the rule before, was 10% slower on average over the random ones; us before
// and after: FP16 256x256x1024 1859 -> 1566; FP32 64x64x128 30.6 -> 24.6;
// 96^3 46.5 -> 36.3; 128^3 87.1 -> 78.3; 128x128x512 unchanged.
inline int pick_zchunk(int tiles, int nzi, int sms, int per_sm) {
    int best = nzi;
    double least = 1e300;
    for (int chunks = 1; chunks <= nzi; ++chunks) {
        const int zc = (nzi + chunks - 1) / chunks;
        if (zc < 2 && nzi >= 2) break;
        const long long n = 1ll * tiles * ((nzi + zc - 1) / zc), slots = 1ll * sms * per_sm;
        double t = double(n / slots) * (zc + 1);
        const long long rem = n % slots;
        if (rem > 0) {
            const int on = int((rem + sms - 1) / sms);  // CTAs on the fullest SM
            t += (per_sm > 1 ? 0.75 + 0.25 * (on - 1) / (per_sm - 1) : 1.0) * (zc + 1) + (on < per_sm ? 4 : 0);
        }
        if (t < least) least = t, best = zc;
    }
    return std::max(best, 1);
}
}  // namespace pflbm
