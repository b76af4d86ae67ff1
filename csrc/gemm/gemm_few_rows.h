// When the few-rows GEMM (gemm_tcgen05_skinny.cu) is taken and how it is launched; plain C++ without CUDA.
#ifndef TILEXR_GEMM_FEW_ROWS_H
#define TILEXR_GEMM_FEW_ROWS_H

#include <algorithm>
#include <cstdint>

namespace TileXR {

constexpr int GEMM_SKINNY_MAX_SPLIT = 8;           // CTAs of a cluster that share a tile's K
constexpr int GEMM_SKINNY_MAX_GROUPS = 256;        // groups of one launch

// Few rows, or few 256 x 256 tiles: the kernel whose tiles are 128 columns by up to 128 rows and which splits K.
// A wide tile takes about 0.005 us per element of K, however few rows it has; the few-rows kernel takes 8 us (16 rows) to 16 us
// (128 rows) before K and N count, and where the columns fill the chip a step of K of a tile of many rows costs it more.
// us, wide and few-rows, weights from memory (n x k):
//    16 rows     8192 x 256    7.1   7.6     16384 x 256    8.4   8.4     16384 x 1024  14.5  13.5     65536 x 4096  94.3  91.1
//    32 rows    16384 x 256    8.3  10.4      8192 x 512    9.1  12.3     16384 x 1024  14.7  15.3     32768 x 4096  51.7  51.5
//    64 rows     8192 x 2048  18.6  16.9     16384 x 2048  20.5  24.6     16384 x 4096  35.3  35.3     24576 x 4096  41.3  45.0
//   128 rows     8192 x 2048  19.9  23.9      8192 x 4096  32.8  28.9     16384 x 4096  37.2  43.5     32768 x 4096  54.4  63.9
//   tiles, k = 4096: 1024 x 1024 (16 tiles) 29.0 25.1, 256 x 4096 (16) 31.1 28.4; 384 x 4096 (32) 29.0 35.0
inline bool FewRows(int64_t m, int64_t n, int64_t k)
{
    const int64_t squareTiles = ((m + 255) / 256) * ((n + 255) / 256);
    if (m <= 16) return true;
    if (m <= 32) return k >= 1024;
    if (m <= 64) return (k >= 2048 && n <= 8192) || (k >= 4096 && n <= 16384);
    return k >= 4096 && (squareTiles <= 16 || (m <= 128 && n <= 8192));
}

// Rows per tile for `rows` rows: the smallest size that holds them, 128 at most.
inline int FewRowsTile(int64_t rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128; }

// Rows per tile for `rows` rows in `groups` groups whose sizes are on the device.  Tiles of twice the average hold most groups, but a
// group of many rows then takes many tiles: 64 groups of 4096 x 2048, 512 rows, all in one group, 49 us with tiles of 16 rows, 29 with 64
// (38 before there was this kernel); with eight rows each 171 and 167, so larger tiles cost the even case nothing from some 100 rows on.
// Below that the rows themselves weigh: one row in each of 8 groups of 4096 x 4096 48 us with 16, 58 with 64.  128 rows where a group
// holds 64 on average: 64 each 179 us with 64 and 183 with 128, sizes falling as 1 / g 214 and 200; up to 48 on average 64 rows are the safer ones
// (2048 x 1024, 48 on average, all in a quarter of the groups: 37 and 43 us, 36 before).
inline int FewRowsGroupTile(int64_t rows, int64_t groups)
{
    if (rows < 128) return 16;
    if (rows <= 256) return 32;
    return rows < 1024 || rows <= 48 * groups ? 64 : 128;
}

struct FewRowsLaunch {
    int split;          // CTAs of a cluster that share a tile's K
    unsigned grid;      // CTAs
};

// `groups` 0: one product; else the groups of all launches.  `tn` rows per tile.  `ctas` caps the CTAs of a launch (0: two on each
// of the `sms` SMs), as it does for the other GEMM kernels: a caller leaves SMs to other work with it.
inline FewRowsLaunch PlanFewRows(int64_t m, int64_t n, int64_t k, int64_t groups, int tn, int sms, int64_t ctas)
{
    const int64_t places = ctas > 0 ? std::min<int64_t>(ctas, 2 * static_cast<int64_t>(sms)) : 2 * static_cast<int64_t>(sms);
    const int64_t items = ((m + tn - 1) / tn + std::min<int64_t>(groups, GEMM_SKINNY_MAX_GROUPS)) * ((n + 127) / 128);
    const int64_t kBlocks = (k + 63) / 64;
    int split = 1;
    if (groups == 0) {
        // K is split while the parts still find a place at once and each keeps four steps of K; no part may be empty
        while (split < GEMM_SKINNY_MAX_SPLIT && items * split * 2 <= places && kBlocks >= split * 2 * 4) split *= 2;
        while (split > 1 && (kBlocks + split - 1) / split * (split - 1) >= kBlocks) split /= 2;
    }
    return {split, static_cast<unsigned>(split > 1 ? items * split : std::max<int64_t>(1, std::min(items, places)))};
}

// How the 256 x 256 tiles of a plain block-scaled fp8 product are dealt out to CTA pairs (the fused forms keep to whole ones: with peers slices were
// not measured): the first `wide` whole, the others in slices of `width` columns, so that a last wave of a few tiles, or a product of a
// few tiles, does not leave most pairs without work.  A slice reads its tile's rows of A again and waits for the same round trips per
// block of K, so a narrow one takes about 0.70 (32 columns), 0.72 or 0.77 (128) of a whole tile at any K from 512 to 8192: the narrowest slices
// that all find a pair at once, and whole tiles where not even those of 128 columns do.
// us at K 2048 on 74 pairs, whole tiles, slices of 128, 64 and 32 columns: 2 tiles 12.1 9.7 9.2 8.8; 16 12.5 10.0 9.4 14.9; 28 12.9 10.3 15.5 26.2;
// 40 13.3 16.7 21.4 31.9; 76 22.4 20.2 19.6 19.5; 224 41.7 39.2 38.7 38.6.  At K 4096, 224 and 448 tiles: 70.3 whole and 64.9 in
// slices of 32, 122.3 and 119.6.
struct Fp8Slices {
    int wide, width, items;
};
inline Fp8Slices PlanFp8Slices(int64_t tiles, int64_t pairs)
{
    const int64_t wide = tiles / pairs * pairs, rest = tiles - wide;
    for (int width = 32; rest > 0 && width <= 128; width *= 2) {
        const int64_t slices = rest * (256 / width);
        if (slices <= pairs) return {static_cast<int>(wide), width, static_cast<int>(wide + slices)};
    }
    return {static_cast<int>(tiles), 256, static_cast<int>(tiles)};
}

// Blocks of the copy in front of a gathered product on one rank: four 16-byte vectors per thread until there are four blocks to an SM, and no more
// than `ctas`, the caller's cap (0: none).
inline int64_t StageCopyBlocks(int64_t vecs, int64_t sms, int64_t ctas)
{
    return std::min((vecs + 1023) / 1024, ctas > 0 ? std::min(ctas, 4 * sms) : 4 * sms);
}

} // namespace TileXR

#endif // TILEXR_GEMM_FEW_ROWS_H
