// Sizes of the fused stage tail's tiles and of a tile's lists (tail_body), in plain C++ for host code too.
#pragma once

#ifdef __CUDACC__
#define AFAR_HOST_DEVICE __host__ __device__
#else
#define AFAR_HOST_DEVICE
#endif

namespace afar {

constexpr int kTailThreads = 256, kTailBlocks = 4;
constexpr int kTailHalo = 128, kTailExtra = 192, kTailList = 32;  // most of each that a tile may have

// The halo entry that a thread past a tile's `cells` own ones loads ahead.  A tile of fewer than
// kTailThreads - kTailHalo cells (96) leaves more such threads than its lists have entries: those load the
// last entry too, and use nothing of it (a tile has at most kTailHalo halo cells).
AFAR_HOST_DEVICE constexpr int tail_first_halo(const int thread, const int cells) {
  return thread - cells < kTailHalo ? thread - cells : kTailHalo - 1;
}

// Cells of a tile (see tail_cells) of a mesh with at most maxM faces a cell.
AFAR_HOST_DEVICE constexpr int tail_tile_cells(const int maxM, const int cells) {
  return maxM <= 3 ? 192 : cells <= 4096 ? 96 : 152;
}

}  // namespace afar
