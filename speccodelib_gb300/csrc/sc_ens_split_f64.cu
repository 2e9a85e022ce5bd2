// Compiled instances: 2D ensembles, one launch per pass, double arithmetic.
#include "sc_ens_split.cuh"
namespace sc {
template <> cudaError_t ens_split_stage<double>(const CUtensorMap& map, const EnsClass<double>& ec, cudaStream_t s) {
  switch (ec.logn) {
    case 6: return ens_split_stage_n<double, 6>(map, ec, s);
    case 7: return ens_split_stage_n<double, 7>(map, ec, s);
    case 8: return ens_split_stage_n<double, 8>(map, ec, s);
    case 9: return ens_split_stage_n<double, 9>(map, ec, s);
    case 10: return ens_split_stage_n<double, 10>(map, ec, s);
    default: return cudaErrorInvalidValue;
  }
}
template <> int ens_split_tile<double>(int logn) {
  switch (logn) {
    case 6: return EnsSplitCfg<double, 6>::P;
    case 7: return EnsSplitCfg<double, 7>::P;
    case 8: return EnsSplitCfg<double, 8>::P;
    case 9: return EnsSplitCfg<double, 9>::P;
    default: return EnsSplitCfg<double, 10>::P;
  }
}
}  // namespace sc
