// Compiled instances: 2D ensembles, one launch per pass, float arithmetic.
#include "sc_ens_split.cuh"
namespace sc {
template <> cudaError_t ens_split_stage<float>(const CUtensorMap& map, const EnsClass<float>& ec, cudaStream_t s) {
  switch (ec.logn) {
    case 6: return ens_split_stage_n<float, 6>(map, ec, s);
    case 7: return ens_split_stage_n<float, 7>(map, ec, s);
    case 8: return ens_split_stage_n<float, 8>(map, ec, s);
    case 9: return ens_split_stage_n<float, 9>(map, ec, s);
    case 10: return ens_split_stage_n<float, 10>(map, ec, s);
    default: return cudaErrorInvalidValue;
  }
}
template <> int ens_split_tile<float>(int logn) {
  switch (logn) {
    case 6: return EnsSplitCfg<float, 6>::P;
    case 7: return EnsSplitCfg<float, 7>::P;
    case 8: return EnsSplitCfg<float, 8>::P;
    case 9: return EnsSplitCfg<float, 9>::P;
    default: return EnsSplitCfg<float, 10>::P;
  }
}
}  // namespace sc
