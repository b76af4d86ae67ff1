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
// (128 rows) before K and N count.  us, wide and few-rows: 1 x 4096 x 1024 (m, n, k) 10.5 and 8.4; 17 x 7168 x 2048 18.4 and 12.3;
// 64 x 4096 x 1024 10.5 and 12.4, x 4096 24.8 and 16.2; 64 x 7168 x 2048 16.6 both, 64 x 16384 x 2048 16.6 and 20.7;
// 128 x 2048 x 2048 16.6 and 17.5, 128 x 7168 x 4096 26.9 and 25.0, 128 x 8192 x 8192 57.6 and 40.2; 512 x 2048 x 4096
// (16 tiles) 29.1 and 27.3, 384 x 4096 x 4096 (32 tiles) 29.0 and 35.0, 512 x 2048 x 2048 18.7 and 22.8.
inline bool FewRows(int64_t m, int64_t n, int64_t k)
{
    const int64_t squareTiles = ((m + 255) / 256) * ((n + 255) / 256);
    return m <= 32 || (m <= 64 && k >= 2048 && n <= 8192) || (k >= 4096 && (m <= 128 || squareTiles <= 16));
}

// Rows per tile for `rows` rows: the smallest size that holds them, 128 at most.
inline int FewRowsTile(int64_t rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128; }

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

} // namespace TileXR

#endif // TILEXR_GEMM_FEW_ROWS_H
