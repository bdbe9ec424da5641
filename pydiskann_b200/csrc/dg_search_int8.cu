// int8-code beam search instantiations (Int8Quantizer, src/sq.rs:121-233).
#include "dg_launch.cuh"
namespace dg {
DgStatus launch_search_int8(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                            bool filt, cudaStream_t st, LaunchInfo *info) {
  (void)lpr;  // tensor-core tiles: no lanes-per-row choice
  return launch_met<TRAV_INT8, 1>(a, Ly, met, cta, tc, filt, st, info);
}
}  // namespace dg
