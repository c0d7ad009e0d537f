// What the search by transforms (search_fft.cu) takes from the shared-product search (search_tile.cu):
// the per-position and per-subset tables, the FP64 refit and the tile kernel's time.
#pragma once
#include "kernels.h"
#include "search_common.cuh"

namespace aldic {

struct SearchTables {
  const float* map;      // 1 / sqrt of the variance sum of every full window position, row-major; 0: a flat window
  const SubsetPrm* prm;  // per subset
  const float2* ringv;   // per subset: (mean, 1 / sqrt) of the partial windows
  int* best;             // per subset: crop index of the first maximum, -1 where the direct kernel decides
  int* flist;            // those subsets (their number: SearchArgs::left)
  void* rows;            // row spectra
};

size_t search_tables_bytes(const SearchArgs& a, size_t row_bytes);
// Fills the tables in a.scratch (the last three are the caller's to write).  Returns the launches.
int launch_search_tables(const SearchArgs& a, size_t row_bytes, SearchTables* t, cudaStream_t st);
void launch_search_refit(const SearchArgs& a, const SearchTables& t, cudaStream_t st);
double search_tile_us(const SearchArgs& a);  // estimate of the tile kernel's time; < 0 without one

}  // namespace aldic
