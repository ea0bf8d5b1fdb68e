// Band storage shared by the batched panels (panels.cu) and the row-skyline path (skyline.cu): the
// lower band of each panel in 32 x 32 FP64 tiles, column-major within a tile; tile (J, d) holds
// block row J + d of block column J, d = 0 .. bt.
#pragma once
#include <cuda_runtime.h>

struct astro_ctx;

namespace astro_band {

constexpr int TB = 32;  // tile edge
constexpr int TT = TB * TB;

struct PanelMeta {
    long long band;   // first double of the panel's tiles
    long long xUnit;  // rows of the padded right-hand-side layout before this panel (times nrhs)
    int n;            // DOF
    int nbc;          // block columns, ceil(n / 32)
    int bt;           // tiles below the diagonal tile in a block column
    int nfac;         // block columns the factorisation eliminates (nbc; fewer for a partial factor)
    int bw;           // entries (i, j) with i - j > bw are zero
    int pad;
};

__device__ __forceinline__ size_t tile_off(const PanelMeta &M, int J, int d) {
    return (size_t)M.band + ((size_t)J * (M.bt + 1) + d) * TT;
}

}  // namespace astro_band

// FP64 band LDL^T of the panels listed in sched by worker (schedPtr), workers clusters of cs CTAs
// (1, 2, 4, 8 or 16) on stream s; *status gets 1 + the number of a panel with a zero or non-finite
// pivot (panels.cu).
cudaError_t band_ldl64(const astro_band::PanelMeta *meta, const int *sched, const int *schedPtr, int workers, int cs,
                       double *band, int *status, cudaStream_t s);
